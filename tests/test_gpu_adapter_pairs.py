"""The adapter backward with two blocks to a 64-row tile (as many rows as give every block an SM of its own) and, one tile
past that line, with blocks that walk: a single tile, ragged last tiles, against float64; the same bits
run to run.  768 wide: the only sites that are planned onto that kernel.  Its bound: every term within 2^-17 of itself (two bf16 pieces of the streamed operand), with
errors of either sign, so 2e-6 of 1 + sum|a_k b_k| once a sum has a few hundred terms; dB and dA sum M of them."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op


@pytest.mark.parametrize("M", [64, 100, 1000, 4699, 4736, 4737])
def test_site_gradients_against_float64(M):
    N, K, r, s = 768, 768, 16, 2.0
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    x = a.alloc(M * K, "normal"); dy = a.alloc(M * N, "normal")
    Bm = a.alloc(r * N, "normal", scale=0.05); t = a.alloc(M * r, "normal")
    dt = a.alloc(M * r); gB = a.alloc(r * N); gA = a.alloc(K * r)
    prog = [
        P.Instr(Op.GEMM_NT, 0, P.f32_bits(s), (dy, Bm, dt, P.NULL_REF), (M, r, N)),
        P.Instr(Op.GEMM_TN, 0, P.f32_bits(s), (t, dy, gB, P.NULL_REF), (r, N, M)),
        P.Instr(Op.GEMM_TN, 0, 0, (x, dt, gA, P.NULL_REF), (K, r, M)),
    ]
    arena0, ro = a.build()

    def run():
        arena = arena0.copy()
        be = B.CudaBackend(0)
        be.set_coherence(B.COHERENCE_LAZY)
        be.bind(arena, ro)
        be.set_program(prog)
        be.run(None)
        be.host_needs(0, arena.size)
        be.flush()
        fused = be.counters().fused_dispatches
        be.close()
        return arena, fused

    def f(arena, off, rows, cols):
        return arena[off:off + 4 * rows * cols].view(np.float32).reshape(rows, cols).astype(np.float64)

    one, fused = run()
    two, _ = run()
    assert np.array_equal(one, two)
    assert fused == 2
    X, DY, BB, T = f(arena0, x, M, K), f(arena0, dy, M, N), f(arena0, Bm, r, N), f(arena0, t, M, r)
    DT = f(one, dt, M, r)
    for name, got, want, mag in (("dT", DT, s * DY @ BB.T, s * np.abs(DY) @ np.abs(BB.T)),
                                 ("dB", f(one, gB, r, N), s * T.T @ DY, s * np.abs(T.T) @ np.abs(DY)),
                                 ("dA", f(one, gA, K, r), X.T @ DT, np.abs(X.T) @ np.abs(DT))):
        assert (np.abs(got - want) / (1.0 + mag)).max() < (2e-6 if name == "dT" or M >= 500 else 2.0 ** -17), name


def test_dt_has_the_bits_of_blocks_that_walk():
    """dT of a row is one sum over the row whatever shares its tile: the first rows of a batch that walks, alone."""
    N, K, r, M = 768, 768, 16, 4800
    rng = np.random.default_rng(5)
    x, dy, t = (rng.standard_normal((M, n)).astype(np.float32) for n in (K, N, r))
    Bm = (rng.standard_normal((r, N)) * 0.05).astype(np.float32)

    def run(rows):
        a = Arena(rng)
        refs = [a.alloc(v.size, v) for v in (x[:rows], dy[:rows], t[:rows], Bm)]
        dt, gB, gA = a.alloc(rows * r), a.alloc(r * N), a.alloc(K * r)
        arena, ro = a.build()
        be = B.CudaBackend(0)
        be.set_coherence(B.COHERENCE_LAZY)
        be.bind(arena, ro)
        be.set_program([
            P.Instr(Op.GEMM_NT, 0, P.f32_bits(2.0), (refs[1], refs[3], dt, P.NULL_REF), (rows, r, N)),
            P.Instr(Op.GEMM_TN, 0, P.f32_bits(2.0), (refs[2], refs[1], gB, P.NULL_REF), (r, N, rows)),
            P.Instr(Op.GEMM_TN, 0, 0, (refs[0], dt, gA, P.NULL_REF), (K, r, rows)),
        ])
        be.run(None)
        be.host_needs(0, arena.size)
        be.flush()
        assert be.counters().fused_dispatches == 2
        be.close()
        return arena[dt:dt + 4 * rows * r].view(np.float32).reshape(rows, r).copy()

    whole = run(M)
    for rows in (64, 1000, 4096):
        assert np.array_equal(run(rows), whole[:rows])
