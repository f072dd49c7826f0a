"""Exact products whose activation is cut into bf16 pieces inside the kernel (a single round of tiles, A row by row):
edges of the 128-row tiles, the column tiles and the 64-wide blocks of K, reductions shared by a cluster, ragged widths,
rows of A off the 16-byte grid's multiples, f32 and int8 weights with every epilogue, operands that are not finite; and
each kernel of the form, bf16 weights among them."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_gpu_umma import bf16_round
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op


def _run(prog, arena0, ro, mode):
    arena = arena0.copy()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.set_split_gemm(mode)
    be.bind(arena, ro)
    be.run(prog)
    be.host_needs(0, arena.size)
    be.flush()
    taken = be.counters().split_executions
    be.close()
    return arena, taken


SHAPES = [(1023, 256, 256), (4096, 256, 256), (129, 1024, 1021), (640, 514, 320), (300, 5000, 256), (4096, 192, 1000), (2000, 385, 96)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("bad", [False, True], ids=["finite", "infinite"])
def test_against_double(shape, bad):
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    x = a.alloc(M * K, "normal"); d = a.alloc(M * N, "normal")
    w = rng.standard_normal(K * N).astype(np.float32)
    q = rng.integers(-127, 128, size=K * N, dtype=np.int8)
    rw, rq = a.ro_alloc(w), a.ro_alloc(q)
    sc, ks = (rng.random(N) * 0.01 + 1e-3).astype(np.float32), (rng.random(K) * 0.01 + 1e-3).astype(np.float32)
    rs, rk = a.ro_alloc(sc), a.ro_alloc(ks)
    bias = rng.standard_normal(N).astype(np.float32)
    rb = a.ro_alloc(bias)
    outs = [a.alloc(M * N) for _ in range(4)]
    dims, f = (M, N, K), P.f32_bits
    prog = [
        P.Instr(Op.GEMM_NN, P.FLAG_EPILOGUE_BIAS | (P.ACT_RELU << 1), f(0.5), (x, rw, outs[0], rb), dims),
        P.Instr(Op.GEMM_NT, P.FLAG_GEMM_ADDEND, f(2.0), (x, rw, outs[1], d), dims),
        P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, rq, outs[2], rs), dims),
        P.Instr(Op.GEMM_NT_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, rq, outs[3], rk), dims),
    ]
    arena, ro = a.build()
    A = arena[x:x + 4 * M * K].view(np.float32).reshape(M, K)
    if bad:
        A[M // 2, K // 3] = np.inf
    got, taken = _run(prog, arena, ro, -1)
    assert taken >= 2
    D = arena[d:d + 4 * M * N].view(np.float32).reshape(M, N).astype(np.float64)
    A64 = A.astype(np.float64)
    wn, wt, qn, qt = (m.astype(np.float64) for m in (w.reshape(K, N), w.reshape(N, K).T, q.reshape(K, N), q.reshape(N, K).T))
    with np.errstate(invalid="ignore"):
        want = [np.maximum(0.5 * (A64 @ wn) + bias, 0), D + 2.0 * (A64 @ wt), (A64 @ qn) * sc, (A64 * ks) @ qt]
    for k, (off, ref) in enumerate(zip(outs, want)):
        g = got[off:off + 4 * M * N].view(np.float32).reshape(M, N).astype(np.float64)
        rows = np.ones(M, bool)
        if bad:
            rows[M // 2] = False
            assert not np.isfinite(g[M // 2]).all()
        # (1.5 + 0.3 sqrt(K / 64)) 2^-24 of the product's root mean square, eight times that at the worst element
        rms = np.sqrt(np.mean(ref[rows] ** 2))
        err = np.abs(g[rows] - ref[rows])
        assert np.sqrt(np.mean(err ** 2)) <= 4e-7 * rms, k
        assert err.max() <= 8e-6 * rms, k


# Each kernel of the form, by the planner's choice on 148 SMs: (M, N, K), weight, the tile width and the CTAs that share a
# tile's K.
FORMS = [
    ((4096, 256, 256), "f32", 64, 1), ((1023, 256, 256), "f32", 64, 4), ((600, 2048, 512), "f32", 128, 1),
    ((256, 4096, 512), "f32", 128, 2), ((640, 514, 320), "f32", 128, 4),
    ((2000, 385, 96), "int8", 64, 1), ((128, 1024, 1024), "bf16", 64, 4), ((300, 5000, 256), "bf16", 128, 1),
    ((4096, 256, 256), "int8", 128, 2), ((640, 514, 320), "bf16", 128, 4), ((4096, 768, 768), "int8", 192, 1),
    ((2048, 768, 1024), "bf16", 192, 2), ((1000, 768, 3072), "int8", 192, 4), ((600, 2048, 512), "bf16", 192, 2),
    # ... where a CTA sums its blocks in two parts, or in four
    ((512, 3072, 320), "f32", 128, 1), ((300, 2048, 640), "f32", 128, 2), ((600, 1024, 320), "f32", 64, 1),
    ((1024, 2048, 1088), "int8", 128, 1), ((512, 2048, 1000), "bf16", 128, 2),
]


@pytest.mark.parametrize("form", FORMS, ids=["%dx%dx%d-%s-w%d-c%d" % (*f[0], *f[1:]) for f in FORMS])
def test_each_kernel_of_the_form(form):
    (M, N, K), kind, _, _ = form
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    x = a.alloc(M * K, "normal")
    out = a.alloc(M * N)
    if kind == "int8":
        w = rng.integers(-127, 128, size=(K, N), dtype=np.int8)
        scale = (rng.random(N) * 0.01 + 1e-3).astype(np.float32)
        ins = P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, a.ro_alloc(w), out, a.ro_alloc(scale)), (M, N, K))
        w64 = w.astype(np.float64) * scale
    else:
        w = rng.standard_normal((K, N)).astype(np.float32)
        if kind == "bf16":
            w = bf16_round(w.reshape(-1)).reshape(K, N)
        stored = (w.view(np.uint32) >> 16).astype(np.uint16) if kind == "bf16" else w
        ins = P.Instr(Op.GEMM_NN_BF16 if kind == "bf16" else Op.GEMM_NN, 0, 0, (x, a.ro_alloc(stored), out, P.NULL_REF), (M, N, K))
        w64 = w.astype(np.float64)
    arena0, ro = a.build()
    A = arena0[x:x + 4 * M * K].view(np.float32).reshape(M, K)
    bad_row, bad_k = M - 1, K // 3
    finite = A.copy()
    A[bad_row, bad_k] = np.inf
    arena = arena0.copy()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(arena, ro)
    be.set_program([ins])
    results, launches = [], []
    for _ in range(3):
        be.run(None)
        be.host_needs(out, 4 * M * N)
        be.flush()
        launches.append(be.counters().kernel_launches)
        results.append(arena[out:out + 4 * M * N].view(np.float32).reshape(M, N).copy())
    assert be.counters().split_executions == 3
    be.close()
    # the weight's pieces are made once; a matrix of A's pieces would be a launch of its own each time
    assert launches[2] - launches[1] == launches[1] - launches[0] == 1
    assert np.array_equal(results[0], results[1], equal_nan=True) and np.array_equal(results[1], results[2], equal_nan=True)
    got = results[0].astype(np.float64)
    with np.errstate(invalid="ignore"):
        assert np.array_equal(results[0][bad_row], (np.inf * w64[bad_k]).astype(np.float32), equal_nan=True)
    want = finite.astype(np.float64)[:bad_row] @ w64
    rms = np.sqrt(np.mean(want ** 2))
    err = np.abs(got[:bad_row] - want)
    assert np.sqrt(np.mean(err ** 2)) <= 4e-7 * rms and err.max() <= 8e-6 * rms   # as above


def test_pieces_that_are_there_are_used_on_a_long_walk():
    """A wide product cuts the activation into a piece matrix; the narrow one after it, which would cut it inside its
    kernel, takes that."""
    M, K = 2048, 2048
    rng = np.random.default_rng(11)
    a = Arena(rng)
    x = a.alloc(M * K, "normal")
    prog, want = [], []
    for N in (2048, 512):
        w = rng.integers(-127, 128, size=(K, N), dtype=np.int8)
        scale = (rng.random(N) * 0.01 + 1e-3).astype(np.float32)
        out = a.alloc(M * N)
        prog.append(P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, a.ro_alloc(w), out, a.ro_alloc(scale)), (M, N, K)))
        want.append((out, N, w * scale.astype(np.float64)))
    arena, ro = a.build()
    A = arena[x:x + 4 * M * K].view(np.float32).reshape(M, K).astype(np.float64)
    both, taken = _run(prog, arena, ro, -1)
    alone, _ = _run(prog[1:], arena, ro, -1)
    assert taken == 2
    for got, (out, N, w) in ((both, want[0]), (both, want[1]), (alone, want[1])):
        ref = A @ w
        err = np.abs(got[out:out + 4 * M * N].view(np.float32).reshape(M, N) - ref)
        rms = np.sqrt(np.mean(ref ** 2))
        assert np.sqrt(np.mean(err ** 2)) <= 4e-7 * rms and err.max() <= 8e-6 * rms


# Scales along k (they join the activation): each tile width, K that ends inside a block, a CTA's part of K that begins inside
# the scales.
SCALED = [(4096, 256, 256), (300, 5000, 256), (4096, 768, 768), (1000, 768, 3072), (640, 514, 328), (129, 1000, 1000), (2000, 385, 96)]


@pytest.mark.parametrize("shape", SCALED, ids=["x".join(map(str, s)) for s in SCALED])
def test_scales_along_k(shape):
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    x, out = a.alloc(M * K, "normal"), a.alloc(M * N)
    q = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
    scale = np.exp2(rng.uniform(-12, -2, size=K)).astype(np.float32)
    prog = [P.Instr(Op.GEMM_NT_Q8, P.FLAG_Q8_COL_SCALE, 0, (x, a.ro_alloc(q.reshape(-1)), out, a.ro_alloc(scale)), (M, N, K))]
    arena, ro = a.build()
    got, taken = _run(prog, arena, ro, -1)
    assert taken == 1
    A = arena[x:x + 4 * M * K].view(np.float32).reshape(M, K)
    want = (A.astype(np.float64) * scale) @ q.T.astype(np.float64)
    err = got[out:out + 4 * M * N].view(np.float32).reshape(M, N) - want
    # (as above, and a rounding of every scaled element)
    assert np.sqrt(np.mean(err ** 2)) <= 4e-7 * np.sqrt(np.mean(want ** 2))
    assert np.abs(err).max() <= 8e-6 * np.sqrt(np.mean(want ** 2))
