"""The rank-r expand product at the edges of its blocks (8 rows, 256 columns) in both orders, with and without a bias and an
activation: bit for bit the CPU's through the strict seam."""

import numpy as np
import pytest

import oracle
from see_ai_b200 import backend as B
from see_ai_b200 import plan as P

pytestmark = pytest.mark.gpu
Op = P.Op


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


@pytest.mark.parametrize("rank", [4, 8, 12, 16])
@pytest.mark.parametrize("M,N", [(64, 64), (65, 68), (71, 260), (72, 256), (130, 1028), (1000, 516)])
def test_expand_matches_the_cpu(M, N, rank):
    rng = np.random.default_rng(M * N + rank)
    sizes = dict(t=M * rank, w=rank * N, bias=N, c0=M * N, nn=M * N, nt=M * N, act=M * N)
    refs, size = {}, 0
    for name, n in sizes.items():
        refs[name] = size
        size += (4 * n + 63) // 64 * 64
    arena = np.zeros(size, dtype=np.uint8)
    for name in ("t", "w", "bias", "c0"):
        arena[refs[name]:refs[name] + 4 * sizes[name]] = rng.standard_normal(sizes[name], dtype=np.float32).view(np.uint8)
    o = refs
    prog = [P.Instr(Op.GEMM_NN, P.FLAG_GEMM_ADDEND, P.f32_bits(2.0), (o["t"], o["w"], o["nn"], o["c0"]), (M, N, rank)),
            P.Instr(Op.GEMM_NT, P.FLAG_GEMM_ADDEND, P.f32_bits(0.5), (o["t"], o["w"], o["nt"], o["c0"]), (M, N, rank)),
            P.Instr(Op.GEMM_NN, P.FLAG_EPILOGUE_BIAS | (1 << P.FLAG_ACT_SHIFT), 0,   # (ReLU)
                    (o["t"], o["w"], o["act"], o["bias"]), (M, N, rank))]
    cpu, gpu = arena.copy(), arena.copy()
    ref = oracle.OracleExecutor()
    ref.bind(cpu, None)
    ref.run(prog, None)
    be = B.CudaBackend(0)
    be.bind(gpu, None)
    be.run(prog, None)
    be.close()
    np.testing.assert_array_equal(gpu, cpu)
