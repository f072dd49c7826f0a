"""Exact products with too few output tiles to fill the GPU, through the strict seam:
the CPU's bits for every form and weight type, at the edges of the 16- and 32-wide
tiles, of the 128-wide k slices and of the quads and lanes inside them."""

import numpy as np
import pytest

import oracle
from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op

SHAPES = [(1, 1, 1), (16, 16, 128), (17, 15, 129), (57, 10, 784), (3, 130, 127), (64, 33, 131), (400, 420, 37), (385, 384, 260)]


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_bits_of_the_cpu_executor(shape):
    M, N, K = shape
    rng = np.random.default_rng(M + 5 * N + 11 * K)
    a = Arena(rng)
    A = a.alloc(M * K, "normal"); At = a.alloc(K * M, "normal"); Bm = a.alloc(K * N, "normal"); Bt = a.alloc(N * K, "normal")
    D = a.alloc(M * N, "normal"); acc = a.alloc(M * N, "normal")
    q = rng.integers(-127, 128, size=K * N, dtype=np.int8)
    h = (rng.standard_normal(N * K).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    rq, rh = a.ro_alloc(q), a.ro_alloc(h)
    rcs = a.ro_alloc((rng.random(N) * 0.02 + 1e-3).astype(np.float32))
    rks = a.ro_alloc((rng.random(K) * 0.02 + 1e-3).astype(np.float32))
    rb = a.ro_alloc(rng.standard_normal(N).astype(np.float32))
    outs = [a.alloc(M * N) for _ in range(6)]
    dims, f = (M, N, K), P.f32_bits
    prog = [
        P.Instr(Op.GEMM_NN, P.FLAG_EPILOGUE_BIAS | (P.ACT_RELU << 1), f(0.5), (A, Bm, outs[0], rb), dims),
        P.Instr(Op.GEMM_NT, P.FLAG_GEMM_ADDEND, f(2.0), (A, Bt, outs[1], D), dims),
        P.Instr(Op.GEMM_TN, 0, f(2.0), (At, Bm, outs[2], P.NULL_REF), dims),
        P.Instr(Op.GEMM_NN_Q8, P.FLAG_Q8_COL_SCALE, 0, (A, rq, outs[3], rcs), dims),
        P.Instr(Op.GEMM_NT_Q8, P.FLAG_Q8_COL_SCALE, 0, (A, rq, outs[4], rks), dims),
        P.Instr(Op.GEMM_NT_BF16, 0, 0, (A, rh, outs[5], P.NULL_REF), dims),
        P.Instr(Op.GEMM_ACC_NN, 0, 0, (A, Bm, acc, f(0.25)), dims),
    ]
    arena, ro = a.build()
    cpu, gpu = arena.copy(), arena.copy()
    ref = oracle.OracleExecutor()
    ref.bind(cpu, ro)
    ref.run(prog)
    be = B.CudaBackend(0)
    be.bind(gpu, ro)
    be.run(prog)
    be.close()
    for name, off in zip(("nn", "nt", "tn", "nn.q8", "nt.q8", "nt.bf16", "acc"), outs + [acc]):
        assert np.array_equal(cpu[off:off + 4 * M * N], gpu[off:off + 4 * M * N]), name
