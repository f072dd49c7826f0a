"""A bias, an activation and an add that follow an exact product are done in its epilogue where nothing else reads the
values in between (lazy coherence): the bits of the separate instructions, fewer launches; and left alone where something does
read them, or the result's place is an operand's."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op

SHAPES = [   # the cut kernel, the piece kernels (one tile, several per SM), the cluster kernel, the kernels in the CPU's order
    (600, 512, 512), (1023, 768, 768), (2048, 3072, 256), (32, 64, 1024), (57, 128, 784), (200, 514, 300), (30, 20, 24),
]


def _run(prog, arena0, ro, fused):
    arena = arena0.copy()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.set_epilogue_fusion(fused)
    be.bind(arena, ro)
    be.run(prog)
    be.host_needs(0, arena.size)
    be.flush()
    c = be.counters()
    be.close()
    return arena, c


def _case(shape, kind, tail, in_place=False, read_between=False, over_operand=False):
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    x, y = a.alloc(M * K, "normal"), a.alloc(M * N, "normal")
    b = a.ro_alloc(rng.standard_normal(N).astype(np.float32))
    z, zb, out, seen = (a.alloc(M * N) for _ in range(4))
    dims = (M, N, K)
    if kind == "f32":
        g = P.Instr(Op.GEMM_NN, 0, P.f32_bits(0.5), (x, a.ro_alloc(rng.standard_normal(K * N).astype(np.float32)), z, P.NULL_REF), dims)
    elif kind == "nt":
        g = P.Instr(Op.GEMM_NT, 0, P.f32_bits(0.5), (x, a.ro_alloc(rng.standard_normal(K * N).astype(np.float32)), z, P.NULL_REF), dims)
    elif kind == "addend":
        g = P.Instr(Op.GEMM_NN, P.FLAG_GEMM_ADDEND, 0, (x, a.ro_alloc(rng.standard_normal(K * N).astype(np.float32)), z, y), dims)
    else:
        q = a.ro_alloc(rng.integers(-127, 128, size=K * N, dtype=np.int8))
        s = a.ro_alloc((rng.random(N) * 0.01 + 1e-3).astype(np.float32))
        g = P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, q, z, s), dims)
    if in_place:
        zb = z
    prog, last = [g], z
    if "b" in tail:
        prog.append(P.Instr(Op.ADD_BIAS, 0, 0, (z, b, zb), (M, N)))
        last = zb
    if read_between:
        prog.append(P.Instr(Op.COPY, 0, 0, (last, seen), (M * N,)))
    if over_operand:
        out = x
    if "g" in tail:
        prog.append(P.Instr(Op.GELU_FWD, 0, 0, (last, out), (M * N,)))
    if "r" in tail:
        prog.append(P.Instr(Op.RELU_FWD, 0, 0, (last, out), (M * N,)))
    if "s" in tail:
        prog.append(P.Instr(Op.SILU_FWD, 0, 0, (last, out), (M * N,)))
    if "+" in tail:
        prog.append(P.Instr(Op.ADD_EW, 0, 0, (y, last, out), (M * N,)))
    # The values in between are overwritten, as a plan's next layer overwrites them.
    final = prog[-1].ins[1 if prog[-1].opcode in (Op.GELU_FWD, Op.RELU_FWD, Op.SILU_FWD) else 2]
    for r in {z, zb} - {final}:
        prog.append(P.Instr(Op.FILL, 0, 0, (r, 0), (M * N, 0, 0)))
    return prog, a.build(), final


@pytest.mark.parametrize("tail", ["bg", "b+", "br", "bs"])
@pytest.mark.parametrize("kind", ["f32", "nt", "q8", "addend"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_the_separate_instructions_bits(shape, kind, tail):
    prog, (arena, ro), _ = _case(shape, kind, tail)
    got, fused = _run(prog, arena, ro, True)
    want, single = _run(prog, arena, ro, False)
    np.testing.assert_array_equal(got, want)
    assert fused.kernel_launches <= single.kernel_launches
    assert fused.fused_dispatches == single.kernel_launches - fused.kernel_launches
    if kind == "q8" and shape == (1023, 768, 768):
        assert fused.fused_dispatches == len(tail)


@pytest.mark.parametrize("shape", [(600, 512, 512), (32, 64, 1024)], ids=["pieces", "clusters"])
@pytest.mark.parametrize("how", ["in_place", "read_between", "over_operand"])
@pytest.mark.parametrize("tail", ["bg", "br"])
def test_values_that_others_read(shape, how, tail):
    M, N, K = shape
    if how == "over_operand" and M * N > M * K:
        pytest.skip("the result does not fit the operand's place")
    prog, (arena, ro), _ = _case(shape, "f32", tail, **{how: True})
    got, fused = _run(prog, arena, ro, True)
    want, single = _run(prog, arena, ro, False)
    np.testing.assert_array_equal(got, want)
    both = {"in_place": 2, "read_between": 1, "over_operand": 1}[how]
    # (a GELU in place of its input, which only the piece kernels take with them, leaves the bias to the others)
    assert fused.fused_dispatches == (min(both, 1) if tail == "bg" and K == 1024 else both)


def sums_that_are_not_finite(shape, kind, tail):
    """An infinity, a NaN, and an overflow of finite operands in the activation: what is remade carries the absorbed bias,
    activation and add.  Returns the counters, absorbed and separate."""
    M, N, K = shape
    prog, (arena, ro), final = _case(shape, kind, tail)
    x = prog[0].ins[0]
    A = arena[x:x + 4 * M * K].view(np.float32).reshape(M, K)
    A[M // 2, K // 3], A[M // 3, K - 1], A[M - 1] = np.inf, np.nan, 3e38
    got, fused = _run(prog, arena, ro, True)
    want, single = _run(prog, arena, ro, False)
    g, w = (a[final:final + 4 * M * N].view(np.float32) for a in (got, want))
    assert not np.isfinite(w).all()
    np.testing.assert_array_equal(g, w)   # (any NaN is as good as another)
    return fused, single


@pytest.mark.parametrize("tail", ["bs", "bg", "b+"])
@pytest.mark.parametrize("kind", ["f32", "q8"])
@pytest.mark.parametrize("shape", [(600, 512, 512), (1023, 768, 768), (200, 514, 304)], ids=["cut", "cut192", "ragged"])
def test_sums_that_are_not_finite(shape, kind, tail):
    fused, single = sums_that_are_not_finite(shape, kind, tail)
    assert fused.fused_dispatches == len(tail) == single.kernel_launches - fused.kernel_launches
