"""No GPU needed: the C-ABI library loads, exports every declared symbol, and every kind of fused
program generates CUDA that NVRTC compiles for sm_100a."""
import itertools
import os
import re

import pytest

from ngraph_python_b200 import lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_header_symbols_exported():
    text = open(os.path.join(ROOT, "include", "b200ng.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = set(re.findall(r"\b(b2_[a-z0-9_]+)\s*\(", text))
    assert len(names) >= 10
    raw = lib.raw()
    for n in sorted(names):
        assert hasattr(raw, n), "library does not export %s" % n
    assert lib.raw().b2_version() >= 100


def test_invalid_program_is_rejected():
    ins = [dict(dtype=lib.F32, strides=(0, 0, 1))]
    outs = [dict(dtype=lib.F32, strides=(0, 0, 1), reg=5)]   # undefined register
    prog = lib.make_program((1, 1, 64), ins, [], [("neg", 0, None)], outs, [], lib.REDUCE_NONE)
    with pytest.raises(lib.B200Error, match="undefined register"):
        lib.ew_check(prog)
    outs = [dict(dtype=lib.FLEX16, slot=-1, strides=(0, 0, 1), reg=1)]
    prog = lib.make_program((1, 1, 64), ins, [], [("neg", 0, None)], outs, [], lib.REDUCE_NONE)
    with pytest.raises(lib.B200Error, match="no slot"):
        lib.ew_check(prog)


MODES = [(lib.REDUCE_NONE, (3, 5, 64)), (lib.REDUCE_C, (1, 7, 4096)), (lib.REDUCE_C, (2, 9, 40)),
         (lib.REDUCE_C, (1, 1, 1 << 22)), (lib.REDUCE_B, (2, 33, 256))]


@pytest.mark.parametrize("mode_dims,flex,vec,probe",
                         list(itertools.product(MODES, (0, 1), (0, 1), (0, 1))))
def test_programs_compile(mode_dims, flex, vec, probe):
    mode, (A, B, Cn) = mode_dims
    dt = lib.FLEX16 if flex else lib.F32
    full = (B * Cn, Cn, 1)
    ins = [dict(dtype=dt, slot=0 if flex else -1, strides=full),
           dict(dtype=dt, slot=1 if flex else -1, strides=(0, 0, 1)),     # broadcast over A, B
           dict(dtype=lib.F32, strides=(B, 1, 0))]                        # broadcast over C
    ops = [("mul", 0, 1), ("add", 4, 2), ("tanh", 5, None), ("maximum", 6, 3), ("exp", 7, None)]
    outs = [dict(dtype=dt, slot=2 if flex else -1, strides=full, reg=8)]
    if mode == lib.REDUCE_NONE:
        reds = []
    elif mode == lib.REDUCE_C:
        st = (B, 1, 0)
        reds = [dict(dtype=dt, slot=3 if flex else -1, strides=st, reg=8, redop="sum"),
                dict(dtype=lib.F32, strides=st, reg=7, redop="argmax")]
    else:
        st = (Cn, 0, 1)
        reds = [dict(dtype=dt, slot=3 if flex else -1, strides=st, reg=8, redop="max"),
                dict(dtype=lib.F32, strides=st, reg=7, redop="argmin")]
    if mode == lib.REDUCE_C and Cn == 1 << 22:
        reds = reds[:1]   # the split variant has no arg reductions
    prog = lib.make_program((A, B, Cn), ins, [0.5], ops, outs, reds, mode)
    src = lib.ew_check(prog, vec=bool(vec), probe=bool(probe), want_source=True)
    assert "b2_ew_main" in src
    if mode == lib.REDUCE_C and Cn == 1 << 22:
        assert "b2_ew_finalize" in src


@pytest.mark.parametrize("vec", (0, 1))
@pytest.mark.parametrize("mode", (lib.REDUCE_NONE, lib.REDUCE_C, lib.REDUCE_B))
def test_argument_in_place_is_not_stored_onto_itself(mode, vec):
    """A result that stores an argument as it was read is stored only where the argument lies somewhere
    else; a result in another layout, or of another register, always."""
    A, B, Cn = 2, 6, 64
    full, swapped = (B * Cn, Cn, 1), (Cn, A * Cn, 1)
    ins = [dict(dtype=lib.F32_AT, strides=full), dict(dtype=lib.F32, strides=full)]
    outs = [dict(dtype=lib.F32, strides=full, reg=2), dict(dtype=lib.F32, strides=full, reg=0),
            dict(dtype=lib.F32, strides=swapped, reg=0), dict(dtype=lib.F32, strides=full, reg=1)]
    red = {lib.REDUCE_NONE: [], lib.REDUCE_C: [(B, 1, 0)], lib.REDUCE_B: [(Cn, 0, 1)]}[mode]
    reds = [dict(dtype=lib.F32, strides=st, reg=2, redop="sum") for st in red]
    prog = lib.make_program((A, B, Cn), ins, [], [("mul", 0, 1)], outs, reds, mode)
    src = lib.ew_check(prog, vec=bool(vec), want_source=True)
    assert src.count("const bool put1 = at0 != (const float*)p.out[1];") == 1
    assert re.findall(r"if \(put(\d)\)", src) == ["1"]
    body = src[src.index("b2_ew_main"):]
    stores = [m.start() for m in re.finditer(r"b2_st4_cs\(o1|o1\[\(c", body)]
    assert len(stores) == 1 and body.rindex("if (put1) {", 0, stores[0]) > body.rindex("}", 0, stores[0])
    assert "put" not in lib.ew_check(prog, vec=bool(vec), probe=True, want_source=True).split("b2_ew_main")[1]


@pytest.mark.parametrize("joint", (False, True))
@pytest.mark.parametrize("vec", (0, 1))
@pytest.mark.parametrize("mode", (lib.REDUCE_NONE, lib.REDUCE_C, lib.REDUCE_B))
def test_a_block_finds_its_place_in_one_line(mode, vec, joint):
    """Blocks of a joint launch belong to one program each: nothing but the line that says where a block
    stands may look at the grid, in either form."""
    if joint and mode != lib.REDUCE_NONE:
        return
    dims = (1, 1, 4096) if joint else (2, 6, 4096)
    ins = [dict(dtype=lib.FLEX16, slot=0, strides=(6 * 4096, 4096, 1))]
    outs = [dict(dtype=lib.F32, strides=(6 * 4096, 4096, 1), reg=1)]
    reds = {lib.REDUCE_NONE: [], lib.REDUCE_C: [(6, 1, 0)], lib.REDUCE_B: [(4096, 0, 1)]}[mode]
    reds = [dict(dtype=lib.F32, strides=st, reg=1, redop="sum") for st in reds]
    prog = lib.make_program(dims, ins, [], [("exp", 0, None)], outs, reds, mode)
    src = lib.ew_check(prog, vec=bool(vec), want_source=True, joint=joint)
    main = src[src.index("b2_ew_main"):].split("b2_ew_finalize")[0]
    lines = [line for line in main.splitlines() if "blockIdx" in line or "gridDim" in line]
    assert len(lines) == (2 if joint else 1) and "block_x = " in lines[-1]
    assert not joint or "jobs.first[at_job + 1]) ++at_job" in lines[0]
    assert ("blocks_y = 1" in main) == joint
