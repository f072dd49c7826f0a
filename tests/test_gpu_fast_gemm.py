"""The small and narrow f32 products of engine mode against float64, to the
reference's bound for its GEMMs (2e-6 of 1 + sum|a_k b_k|;
test/runtime/executor/kernels_test.cc:1786-1822), and identical run to run: every
tile shape of the kernel at its edges, reductions shorter than a warp's slice, cut
over one to eight CTAs, ragged by 1 to 3 (4-byte copies), longer than two buffers."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op

SHAPES = [(1, 1, 1), (32, 1024, 256), (32, 64, 1024), (57, 10, 128), (600, 8, 512), (300, 16, 4096), (65, 4, 37), (8, 512, 600),
          (16, 100, 1030), (3, 70, 259), (33, 33, 5), (100, 7, 2049), (48, 1024, 8), (512, 8, 100)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_products_match_float64_and_repeat(shape):
    M, N, K = shape
    rng = np.random.default_rng(M * 31 + N * 17 + K)
    a = Arena(rng)
    A = a.alloc(M * K, "normal"); At = a.alloc(K * M, "normal"); Bm = a.alloc(K * N, "normal"); Bt = a.alloc(N * K, "normal")
    D = a.alloc(M * N, "normal"); bias = a.ro_alloc(rng.standard_normal(N).astype(np.float32))
    outs = [a.alloc(M * N) for _ in range(4)]
    acc = a.alloc(M * N, "normal")
    dims, f = (M, N, K), P.f32_bits
    prog = [
        P.Instr(Op.GEMM_NN, P.FLAG_EPILOGUE_BIAS | (P.ACT_RELU << 1), f(0.5), (A, Bm, outs[0], bias), dims),
        P.Instr(Op.GEMM_NT, P.FLAG_GEMM_ADDEND, f(2.0), (A, Bt, outs[1], D), dims),
        P.Instr(Op.GEMM_TN, 0, f(2.0), (At, Bm, outs[2], P.NULL_REF), dims),
        P.Instr(Op.GEMM_NN, 0, 0, (A, Bm, outs[3], P.NULL_REF), dims),
        P.Instr(Op.GEMM_ACC_NN, 0, 0, (A, Bm, acc, f(0.25)), dims),
    ]
    arena0, ro = a.build()

    def run():
        arena = arena0.copy()
        be = B.CudaBackend(0)
        be.set_coherence(B.COHERENCE_LAZY)
        be.bind(arena, ro)
        be.run(prog)
        be.host_needs(0, arena.size)
        be.close()
        return arena

    got = run()
    assert np.array_equal(got, run())

    def mat(x, off, rows, cols):
        return x[off:off + 4 * rows * cols].view(np.float32).astype(np.float64).reshape(rows, cols)

    Am, Atm, Bmm, Btm, Dm = (mat(arena0, o, r, c) for o, r, c in ((A, M, K), (At, K, M), (Bm, K, N), (Bt, N, K), (D, M, N)))
    bv = np.frombuffer(ro.tobytes()[bias & ~P.RODATA_BIT:(bias & ~P.RODATA_BIT) + 4 * N], np.float32).astype(np.float64)
    mag = np.abs(Am) @ np.abs(Bmm)
    wants = [
        (outs[0], np.maximum(0.5 * (Am @ Bmm) + bv, 0), 0.5 * mag + np.abs(bv)),
        (outs[1], 2.0 * (Am @ Btm.T) + Dm, 2.0 * (np.abs(Am) @ np.abs(Btm.T)) + np.abs(Dm)),
        (outs[2], 2.0 * (Atm.T @ Bmm), 2.0 * (np.abs(Atm.T) @ np.abs(Bmm))),
        (outs[3], Am @ Bmm, mag),
        (acc, mat(arena0, acc, M, N) + 0.25 * (Am @ Bmm), np.abs(mat(arena0, acc, M, N)) + 0.25 * mag),
    ]
    for off, want, scale in wants:
        assert (np.abs(mat(got, off, M, N) - want) / (1.0 + scale)).max() < 2e-6


@pytest.mark.parametrize("shape", [(57, 128, 784), (33, 33, 5), (40, 64, 1030), (300, 260, 512), (600, 512, 768)],
                         ids=lambda s: "x".join(map(str, s)))
def test_split_gemm_0_keeps_the_order_of_the_strict_seam(shape):
    """With the switch off, lazy coherence leaves the bits of the strict seam, which are the CPU's: products of
    every form (nothing here is rank-r), the exact attention chain."""
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    A = a.alloc(M * K, "normal"); At = a.alloc(K * M, "normal"); Bm = a.alloc(K * N, "normal"); Bt = a.alloc(N * K, "normal")
    outs = [a.alloc(M * N) for _ in range(3)]
    Bq, S, H, d = 2, 70, 2, 16
    n = Bq * S * H * d
    q, k, v, do = (a.alloc(n, "normal") for _ in range(4))
    o, dq, dk, dv = (a.alloc(n) for _ in range(4))
    stats = a.alloc(4 * Bq * H * S)
    geo, bs, hd = P.pack_attn_geometry(Bq, S, H, d), P.pack2(Bq, S), P.pack2(H, d)
    prog = [
        P.Instr(Op.GEMM_NN, 0, P.f32_bits(0.5), (A, Bm, outs[0], P.NULL_REF), (M, N, K)),
        P.Instr(Op.GEMM_NT, 0, 0, (A, Bt, outs[1], P.NULL_REF), (M, N, K)),
        P.Instr(Op.GEMM_TN, 0, 0, (At, Bm, outs[2], P.NULL_REF), (M, N, K)),
        P.Instr(Op.ATTN_FWD_TILED, 0, 0, (q, k, v, o), (stats, bs, hd)),
        P.Instr(Op.ATTN_DQ_TILED, 0, 0, (q, k, v, do), (stats, dq, geo)),
        P.Instr(Op.ATTN_DK_TILED, 0, 0, (q, k, v, do), (stats, dk, geo)),
        P.Instr(Op.ATTN_DV_TILED, 0, 0, (q, k, v, do), (stats, dv, geo)),
    ]
    arena0, ro = a.build()

    def run(lazy):
        arena = arena0.copy()
        be = B.CudaBackend(0)
        if lazy:
            be.set_coherence(B.COHERENCE_LAZY)
            be.set_split_gemm(0)
        be.bind(arena, ro)
        be.run(prog)
        be.host_needs(0, arena.size)
        be.close()
        return arena

    assert np.array_equal(run(True), run(False))


@pytest.mark.parametrize("shape", [(16, 768, 8191), (16, 768, 8192), (8, 66, 20001), (768, 16, 16383), (768, 16, 16384), (256, 4, 17000)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gradients_over_many_rows(shape):
    """Both sides of the row counts at which a rank-r factor's gradient goes from clusters to chunks of rows, in a
    run of its own and behind one that needs less scratch; the reference's bound for its GEMMs as above."""
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    At, Bm, C = a.alloc(K * M, "normal"), a.alloc(K * N, "normal"), a.alloc(M * N)
    arena0, ro = a.build()
    big = P.Instr(Op.GEMM_TN, 0, P.f32_bits(2.0), (At, Bm, C, P.NULL_REF), (M, N, K))
    small = P.Instr(Op.GEMM_TN, 0, 0, (At, Bm, C, P.NULL_REF), (M, N, 300))

    def run(progs):
        arena = arena0.copy()
        be = B.CudaBackend(0)
        be.set_coherence(B.COHERENCE_LAZY)
        be.bind(arena, ro)
        for p in progs:
            be.run(p)
        be.host_needs(C, 4 * M * N)
        be.close()
        return arena[C:C + 4 * M * N].view(np.float32).astype(np.float64).reshape(M, N)

    got = run([[big]])
    assert np.array_equal(got, run([[small], [big], [small, big]]))
    x = arena0[At:At + 4 * K * M].view(np.float32).astype(np.float64).reshape(K, M)
    w = arena0[Bm:Bm + 4 * K * N].view(np.float32).astype(np.float64).reshape(K, N)
    assert (np.abs(got - 2.0 * (x.T @ w)) / (1.0 + 2.0 * (np.abs(x).T @ np.abs(w)))).max() < 2e-6
