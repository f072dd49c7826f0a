"""The exact attention family where its bits are not observed (lazy coherence): double dots on the FP64 tensor
instruction, output sums with fused multiply-adds.  At the edges of the tile kernels, instruction by instruction from the
CPU oracle's bytes, to the 1e-5 of each tensor's scale the executor is held to."""

import numpy as np
import pytest

import oracle
from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_gpu_attention_exact import _program
from tests.util import compare

pytestmark = pytest.mark.gpu

SHAPES = [   # B, S, H, d: one, two and four rows per thread; remainders of 8 features, 16 and 64 rows
    (1, 1, 1, 8), (1, 65, 3, 64), (1, 130, 1, 66), (2, 64, 1, 20), (1, 257, 1, 33), (10, 70, 10, 12), (20, 65, 16, 8), (8, 129, 12, 64),
]
FULL_BLOCKS = [(5, 480, 4, 128), (5, 600, 2, 64)]   # score rows and operands that fill what shared memory two blocks of 32 or 16 rows have


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


@pytest.mark.parametrize("segments", [0, 1], ids=["causal", "segments"])
@pytest.mark.parametrize("shape", SHAPES + FULL_BLOCKS, ids=["x".join(map(str, s)) for s in SHAPES + FULL_BLOCKS])
def test_every_instruction_from_the_oracles_bytes(shape, segments):
    prog, arena = _program(*shape, segments, cached=True)
    cpu, gpu = arena.copy(), arena.copy()
    ref = oracle.OracleExecutor()
    ref.bind(cpu, None)
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(gpu, None)
    be.set_program(prog)
    failures = []
    for i, ins in enumerate(prog):
        before = cpu.copy()
        ref.run(prog, None, i, i + 1)
        gpu[:] = before
        be.host_wrote(0, gpu.size)
        be.run(None, None, i, i + 1)
        be.host_needs(0, gpu.size)
        be.flush()
        diff = np.flatnonzero(cpu != gpu)
        if diff.size:
            lo, hi = diff[0] // 4 * 4, diff[-1] // 4 * 4 + 4
            ok, ratio = compare(gpu[lo:hi].tobytes(), cpu[lo:hi].tobytes(), 1e-5, 1e-7)
            if not ok:
                failures.append(f"{P.OP_NAMES[ins.opcode]}: err/bound {ratio:.3g}")
    be.close()
    assert not failures, "\n".join(failures)
