"""A range finds its device tables (adapter matrices to cut, tensors of the optimizer launch) as the last pass uploaded
them, and uploads them again where the program at the same place in memory says something else."""

import ctypes

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from see_ai_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _gemm_program(alpha):
    prog = W.gemm_step_program(256, True, 8)
    prog.instrs[2].imm = P.f32_bits(alpha)   # the expand product that the frozen product's launch absorbs
    return prog


def _adam_program(first):
    """Two runs of AdamW over tensors at offsets that depend on `first`."""
    n = 96
    rng = np.random.default_rng(5)
    arena = rng.standard_normal(16 * n).astype(np.float32)
    arena[12 * n:] = np.abs(arena[12 * n:])   # second moments
    instrs = [P.Instr(P.Op.ADAMW_STEP, 0, 0, (4 * n * (t ^ first), 4 * n * (4 + t), 4 * n * (8 + t), 4 * n * (12 + t)), (n, 0, 0))
              for t in range(4)]
    return instrs, arena.view(np.uint8).copy()


def _fresh(instrs, arena, rodata):
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(arena, rodata)
    be.set_program(P.pack_program(instrs))
    return be


def _result(be, arena):
    be.run()
    be.host_needs(0, arena.size)
    return arena.copy()


def _same_place(programs, arena, rodata):
    """Each program in turn through one backend, at one address; and each through a backend of its own."""
    start = arena.copy()
    be = _fresh(programs[0], arena, rodata)
    buf, _ = be._prog
    for instrs in programs:
        code = P.pack_program(instrs)
        ctypes.memmove(ctypes.addressof(buf), bytes(code), len(bytes(code)))
        for _ in range(2):   # (the second pass finds the table)
            arena[:] = start
            be.host_wrote(0, arena.size)
            got = _result(be, arena)
            other = start.copy()
            own = _fresh(instrs, other, rodata)
            want = _result(own, other)
            own.close()
            np.testing.assert_array_equal(got, want)
    be.close()


def test_adapter_table_follows_the_program():
    progs = [_gemm_program(a) for a in (2.0, 3.0, 2.0)]
    _same_place([p.instrs for p in progs], progs[0].arena, progs[0].rodata)


def test_optimizer_table_follows_the_program():
    programs = [_adam_program(f) for f in (0, 1, 0)]
    _same_place([p[0] for p in programs], programs[0][1], np.zeros(64, dtype=np.uint8))
