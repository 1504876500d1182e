"""Chained kernels (those that start with chain_begin()) run while the kernel
before them still writes states, scalars, slopes, gradients and cotangents.
Only the set-up tables may be read through the read-only path (__ldg or a
const __restrict__ pointer): its loads ask for data that do not change while
the kernel lives, and may move above the wait.  Checked on the sources: every
chained kernel and every device function it calls."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hom3_b200", "csrc")

# what is written at set-up only: grid, condition and halo tables, cell centres, velocities, index maps
TABLE_ARGS = {"xc", "gsrc", "idx"}
TABLE_READS = re.compile(r"^(reinterpret_cast<const \w+\*>\()?"
                         r"(g\.(nbr|lvl|sub|vel)|sg\.(h\.\w+|pack[23])|ch\.(hnb|bsel|blist|h1end)|hg\.\w+|"
                         r"xc|gsrc|idx|slots)\b")
TABLE_FIELDS = {"nbr", "lvl", "sub", "blk_inst", "inst_end", "vel", "bndry", "pos", "bc_apply", "bc_own", "dx", "partner",
                "xc", "ginst", "lnb", "halo_ids", "halo_off", "grp", "grp_off", "h1end", "hnb", "blist", "bsel", "pack3",
                "pack2"}


def _closing(s, i, o, c):
    n = 0
    for j in range(i, len(s)):
        n += (s[j] == o) - (s[j] == c)
        if n == 0 and s[j] == c:
            return j
    raise AssertionError("unbalanced source")


def _functions():
    """name -> [(file, arguments, body)] of the device functions and kernels."""
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        s = re.sub(r"//[^\n]*", "", open(f).read())
        for m in re.finditer(r"__(?:global|device)__[^;{}]*?\b(\w+)\(", s):
            name, i = m.group(1), m.end() - 1
            if name == "__launch_bounds__":
                i = _closing(s, i, "(", ")") + 1
                m2 = re.compile(r"\s*(\w+)\(").match(s, i)
                name, i = m2.group(1), m2.end() - 1
            e = _closing(s, i, "(", ")")
            b = re.compile(r"\s*\{").match(s, e + 1)
            if b:
                out.setdefault(name, []).append((os.path.basename(f), s[i + 1:e],
                                                 s[b.end() - 1:_closing(s, b.end() - 1, "{", "}") + 1]))
    return out


FUNCS = _functions()
CHAINED = sorted(n for n, d in FUNCS.items() if any("chain_begin()" in b for _, _, b in d))


def _reached(name):
    seen, todo = set(), [name]
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for _, _, body in FUNCS[n]:
            todo += [w for w in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", body) if w in FUNCS]
    return seen


def test_the_chained_kernels_are_found():
    assert {"k_stage", "k_stage_scalar", "k_stage_split", "k_stage_cns_halo", "k_ghost_slopes", "k_stage_muscl",
            "k_muscl_grad", "k_slopes", "k_bc", "k_cfl", "k_adj_ausm"} <= set(CHAINED)
    assert "load_prim" in _reached("k_stage_split") and "prim_w" in _reached("k_stage_muscl")


@pytest.mark.parametrize("kernel", CHAINED)
def test_only_tables_are_read_through_the_read_only_path(kernel):
    for name in sorted(_reached(kernel)):
        for f, args, body in FUNCS[name]:
            const = re.findall(r"\bconst\s+\w+(?:\s+\w+)?\s*\*\s*__restrict__\s+(\w+)", args)
            assert set(const) <= TABLE_ARGS, (f, name, const)
            reads = [r for r in re.findall(r"__ldg\(\s*([^;]*)", body) if not TABLE_READS.match(r)]
            assert not reads, (f, name, reads)


def test_only_tables_are_const_restrict_members():
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.hpp"))):
        for m in re.findall(r"^\s*const\s+\w+(?:\s+\w+)?\*\s*__restrict__\s+(\w+);", open(f).read(), re.M):
            assert m in TABLE_FIELDS, (os.path.basename(f), m)
