"""Exact products on the tensor cores in lazy coherence: every shape and weight
type worth a launch, held to the reference's own bound for its GEMMs (2e-6 of
1 + sum|a_k b_k| against a float64 product; reference:
test/runtime/executor/kernels_test.cc:1786-1822).  The shapes cross what the tile
kernel can get wrong: fewer rows than a tile, widths and reductions that are no
multiple of the tile, of 64, of 8 or of 4, reductions cut over a cluster, the
persistent kernel's ragged rows."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op

SHAPES = [(17, 4096, 1024), (37, 1001, 704), (600, 512, 2048), (257, 2003, 520), (128, 129, 1040), (130, 4100, 66),
          (5000, 3001, 72), (3000, 1025, 33)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_products_of_every_weight_type_match_float64(shape):
    M, N, K = shape
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    a = Arena(rng)
    A = a.alloc(M * K, "normal"); At = a.alloc(K * M, "normal"); D = a.alloc(M * N, "normal")
    Bt = a.alloc(N * K, "normal")
    w = rng.standard_normal((K, N)).astype(np.float32)
    q = rng.integers(-127, 128, size=(K, N), dtype=np.int8)
    h = (rng.standard_normal((N, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    cs = (rng.random(N) * 0.02 + 1e-3).astype(np.float32)
    ks = (rng.random(K) * 0.02 + 1e-3).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    rw, rq, rqt, rh = a.ro_alloc(w), a.ro_alloc(q), a.ro_alloc(np.ascontiguousarray(q.T)), a.ro_alloc(h)
    rcs, rks, rb = a.ro_alloc(cs), a.ro_alloc(ks), a.ro_alloc(bias)
    outs = [a.alloc(M * N) for _ in range(6)]
    dims, f = (M, N, K), P.f32_bits
    prog = [
        P.Instr(Op.GEMM_NN, P.FLAG_EPILOGUE_BIAS | (P.ACT_RELU << 1), 0, (A, rw, outs[0], rb), dims),
        P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (A, rq, outs[1], rcs), dims),
        P.Instr(Op.GEMM_NT_Q8, P.FLAG_Q8_COL_SCALE, 0, (A, rqt, outs[2], rks), dims),
        P.Instr(Op.GEMM_NT_BF16, 0, 0, (A, rh, outs[3], P.NULL_REF), dims),
        P.Instr(Op.GEMM_NT, P.FLAG_GEMM_ADDEND, f(0.375), (A, Bt, outs[4], D), dims),
        P.Instr(Op.GEMM_TN, 0, f(2.0), (At, rw, outs[5], P.NULL_REF), dims),
    ]
    arena, ro = a.build()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(arena, ro)
    be.run(prog)
    taken = be.counters().split_executions
    for off in outs:
        be.host_needs(off, 4 * M * N)
    be.close()
    assert taken == (6 if K % 8 == 0 else 3), taken   # (a narrow weight's rows must be 16-byte pitched)

    def mat(off, rows, cols):
        return arena[off:off + 4 * rows * cols].view(np.float32).astype(np.float64).reshape(rows, cols)

    Am, Atm, Dm, Btm = mat(A, M, K), mat(At, K, M), mat(D, M, N), mat(Bt, N, K)
    w, q, h = w.astype(np.float64), q.astype(np.float64), (h.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    absA = np.abs(Am)
    wants = [
        (np.maximum(Am @ w + bias, 0), absA @ np.abs(w) + np.abs(bias)),
        ((Am @ q) * cs, (absA @ np.abs(q)) * cs),
        ((Am * ks) @ q, (absA * ks) @ np.abs(q)),
        (Am @ h.T, absA @ np.abs(h.T)),
        (0.375 * (Am @ Btm.T) + Dm, 0.375 * (absA @ np.abs(Btm.T)) + np.abs(Dm)),
        (2.0 * (Atm.T @ w), 2.0 * (np.abs(Atm.T) @ np.abs(w))),
    ]
    worst = [float((np.abs(mat(off, M, N) - want) / (1.0 + mag)).max()) for off, (want, mag) in zip(outs, wants)]
    assert max(worst) < 2e-6, worst
