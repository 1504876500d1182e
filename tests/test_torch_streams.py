"""CUDA tensors handed to a solver: its stream is not torch's, so the call waits for torch's current stream before the
library sees the address (the tensor's contents, and the earlier users of its memory)."""
import numpy as np
import pytest
import torch

from hom3_b200 import solver as S


class _Tensor:
    is_cuda, dtype, shape = True, torch.float64, (4, 8)

    def __init__(self, log, device):
        self.log, self.index = log, device

    def contiguous(self):
        self.log.append("copy")
        return self

    def is_contiguous(self):
        return True

    def get_device(self):
        return self.index

    def data_ptr(self):
        return 4096


class _Stream:
    def __init__(self, log):
        self.log = log

    def synchronize(self):
        self.log.append("synchronize")


class _Lib:
    def __init__(self, log):
        self.log = log

    def __getattr__(self, name):
        return lambda *a: self.log.append(name if name != "h3c_wait_stream" else (name, a[1])) or 0


@pytest.mark.parametrize("device", [0, 1])
@pytest.mark.parametrize("call", ["set_state", "state", "adjoint"])
def test_the_solver_waits_for_torchs_stream(call, device, monkeypatch):
    log = []
    monkeypatch.setattr(S, "lib", lambda: _Lib(log))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: _Stream(log))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 77, raising=False)
    monkeypatch.setattr(torch, "empty_like", lambda t: _Tensor(log, device))
    s = S.Solver.__new__(S.Solver)
    s.h, s.nv, s.n_cells = None, 4, 8
    if call == "set_state":
        s.set_state(_Tensor(log, device))
    elif call == "state":
        s.state(out=_Tensor(log, device))
    else:
        s.adjoint(1, _Tensor(log, device))
    name = {"set_state": "h3c_set_state", "state": "h3c_get_state", "adjoint": "h3c_adjoint"}[call]
    wait = ["synchronize" if device else ("h3c_wait_stream", 77)]  # another device's stream is waited for on the host
    copy = [] if call == "state" else ["copy"]  # the copy runs on torch's stream too
    assert log == copy + wait * (2 if call == "adjoint" else 1) + [name]


@pytest.mark.gpu
def test_a_state_still_being_computed_by_torch():
    import cases
    _, (o,) = cases.euler_case("explosion", nd=3, level=4)
    s = cases.gpu_solver_from_oracle(o)
    q = o.state(0)
    a = torch.randn(4096, 4096, device="cuda")
    base = torch.tensor(q, device="cuda")
    out = torch.empty_like(base)
    for i in range(1, 4):
        b = a
        for _ in range(40):
            b = torch.tanh(b @ a)  # some ten ms of work ahead of the state
        t = base * (1.0 + i) + 0.0 * b[:1, :1].double()
        s.set_state(t.t().contiguous().t())  # not contiguous: the solver's own copy comes last on torch's stream
        s.state(out=out)
        assert np.array_equal(out.cpu().numpy()[:, :o.first_ghost], q[:, :o.first_ghost] * (1.0 + i))
