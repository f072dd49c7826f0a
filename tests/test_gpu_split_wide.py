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


def _product(kind, M, N, K, nonneg, coherence):
    """(result, float64 result, sum|a_k b_k|, split executions) of one product."""
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    draw = (lambda *s: np.abs(rng.standard_normal(s)).astype(np.float32)) if nonneg else \
        (lambda *s: rng.standard_normal(s).astype(np.float32))
    a = Arena(rng)
    A = a.alloc(M * K)
    X = draw(*((K, M) if kind == "tn" else (M, K)))
    shape = (N, K) if kind.startswith("nt") else (K, N)
    if kind.endswith("q8"):
        W = rng.integers(0 if nonneg else -127, 128, size=shape, dtype=np.int8)
        scale = (rng.random(K if kind == "ntq8" else N) * 0.02 + 1e-3).astype(np.float32)
        flags, last, op = P.FLAG_Q8_COL_SCALE, a.ro_alloc(scale), Op.GEMM_NT_Q8 if kind == "ntq8" else Op.GEMM_NN_Q8
    else:
        W, flags, last, op = draw(*shape), 0, P.NULL_REF, dict(nn=Op.GEMM_NN, nt=Op.GEMM_NT, tn=Op.GEMM_TN)[kind]
    C = a.alloc(M * N)
    ins = P.Instr(op, flags, 0, (A, a.ro_alloc(W), C, last), (M, N, K))
    arena, ro = a.build()
    arena[A:A + X.nbytes] = X.reshape(-1).view(np.uint8)
    be = B.CudaBackend(0)
    be.set_coherence(coherence)
    be.bind(arena, ro)
    be.run([ins])
    taken = be.counters().split_executions
    be.host_needs(C, 4 * M * N)
    be.close()
    x, w = X.astype(np.float64), W.astype(np.float64)
    x, w = (x.T if kind == "tn" else x), (w.T if kind.startswith("nt") else w)
    if kind == "nnq8":
        w = w * scale
    if kind == "ntq8":
        x = x * scale
    return arena[C:C + 4 * M * N].view(np.float32).astype(np.float64).reshape(M, N), x @ w, np.abs(x) @ np.abs(w), taken


@pytest.mark.parametrize("kind", ["nn", "nt", "tn", "nnq8", "ntq8"])
@pytest.mark.parametrize("shape", [(384, 640, 256), (1000, 768, 768), (600, 768, 3072), (4096, 3072, 256), (300, 256, 8192)],
                         ids=lambda s: "x".join(map(str, s)))
def test_no_further_from_float64_than_the_cuda_core_sums(kind, shape):
    """The tensor core truncates at its accumulator's magnitude; blocks of 64 meet in rounded f32 sums so that
    the whole is as accurate as the kernels in the reference's order, whatever K (rms over the output, 5 % for
    the spread of a sample)."""
    got, want, _, taken = _product(kind, *shape, False, B.COHERENCE_LAZY)
    ref, _, _, none = _product(kind, *shape, False, B.COHERENCE_STRICT)
    assert (taken, none) == (1, 0)
    err, bar = np.sqrt(np.mean((got - want) ** 2)), np.sqrt(np.mean((ref - want) ** 2))
    assert err <= 1.05 * bar, err / bar


@pytest.mark.parametrize("kind", ["nn", "nt", "tn", "nnq8", "ntq8"])
@pytest.mark.parametrize("shape", [(600, 512, 8192), (200, 136, 32000), (2100, 4096, 2048)], ids=lambda s: "x".join(map(str, s)))
def test_same_signed_terms_over_a_long_reduction(kind, shape):
    """Where every term adds up, truncation at the accumulator would grow with K (8e-5 at 32000 over one
    accumulator).  Held to the reference's 2e-6 of sum|a_k b_k|."""
    got, want, mag, taken = _product(kind, *shape, True, B.COHERENCE_LAZY)
    assert taken == 1
    assert (np.abs(got - want) / mag).max() < 2e-6


# A cluster's splits, one tile per SM, ragged widths, the persistent kernel with aligned and ragged rows.
NONFINITE = [(600, 512, 2048), (257, 2003, 520), (4096, 4096, 256), (5000, 3001, 72)]


@pytest.mark.parametrize("kind", ["nn", "nt", "tn", "nnq8", "ntq8"])
@pytest.mark.parametrize("shape", NONFINITE, ids=["x".join(map(str, s)) for s in NONFINITE])
def test_values_no_piece_holds(kind, shape):
    """Infinities, NaNs and finite values above the largest bf16 in an activation (and in an f32 weight) leave what
    the kernels in the reference's order leave: the same infinities and NaNs, finite results to 1e-5 of the row."""
    M, N, K = shape
    rng = np.random.default_rng(M + N)
    a = Arena(rng)
    A, C = a.alloc(M * K), a.alloc(M * N)
    X = rng.standard_normal((M, K)).astype(np.float32)
    X[3, 5], X[M // 2, K - 1], X[M - 1, 0] = np.inf, -np.inf, np.nan
    X[7, 2], X[7, 9] = np.inf, -np.inf
    X[11, :] = 0.0
    X[11, 4] = np.float32(3.4e38)      # finite, above the largest bf16
    shape_w = (N, K) if kind.startswith("nt") else (K, N)
    flags, last = 0, P.NULL_REF
    if kind.endswith("q8"):
        W = rng.integers(-127, 128, size=shape_w, dtype=np.int8)
        W[5 % shape_w[0], 5] = 0       # infinity times zero
        flags, op = P.FLAG_Q8_COL_SCALE, Op.GEMM_NT_Q8 if kind == "ntq8" else Op.GEMM_NN_Q8
        last = a.ro_alloc((rng.random(K if kind == "ntq8" else N) * 0.001 + 1e-3).astype(np.float32))
    else:
        W = (rng.standard_normal(shape_w) * 0.02).astype(np.float32)
        (W if kind.startswith("nt") else W.T)[9, 1] = np.inf
        op = dict(nn=Op.GEMM_NN, nt=Op.GEMM_NT, tn=Op.GEMM_TN)[kind]
    ins = P.Instr(op, flags, 0, (A, a.ro_alloc(W), C, last), (M, N, K))
    arena, ro = a.build()
    arena[A:A + X.nbytes] = (X.T if kind == "tn" else X).reshape(-1).copy().view(np.uint8)

    def run(coherence):
        got = arena.copy()
        be = B.CudaBackend(0)
        be.set_coherence(coherence)
        be.bind(got, ro)
        be.run([ins])
        taken = be.counters().split_executions
        be.host_needs(C, 4 * M * N)
        be.close()
        return got[C:C + 4 * M * N].view(np.float32).astype(np.float64).reshape(M, N), taken

    (got, taken), (want, _) = run(B.COHERENCE_LAZY), run(B.COHERENCE_STRICT)
    assert taken == (0 if kind.endswith("q8") and K % 8 else 1)
    assert not np.isfinite(want).all() and np.isfinite(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    ok = np.isfinite(want)
    scale = np.max(np.abs(np.where(ok, want, 0.0)), axis=1, keepdims=True)
    assert (np.abs(np.where(ok, got, 0.0) - np.where(ok, want, 0.0)) <= 1e-5 * scale).all()


def test_no_piece_buffer_for_products_that_are_refused():
    """An int8 weight whose rows TMA cannot take runs on the CUDA cores: its activation needs no pieces (123 MB)."""
    import torch

    M, N, K = 20000, 256, 1001
    rng = np.random.default_rng(5)
    a = Arena(rng)
    A, C = a.alloc(M * K), a.alloc(M * N)
    rq, rs = a.ro_alloc(rng.integers(-127, 128, size=(K, N), dtype=np.int8)), a.ro_alloc(np.ones(N, np.float32))
    arena, ro = a.build()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(arena, ro)
    be.run([P.Instr(Op.GEMM_NN, 0, 0, (A, A, C, P.NULL_REF), (1, 1, 1))])   # (what a first run allocates)
    before = torch.cuda.mem_get_info(0)[0]
    be.run([P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (A, rq, C, rs), (M, N, K))])
    taken = before - torch.cuda.mem_get_info(0)[0]
    be.close()
    assert taken < 64 << 20, taken
