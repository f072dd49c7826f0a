"""A merge program's deltas as one launch: the bits of the instruction-by-instruction
run, ragged rows and columns and a run longer than one launch's table included, and
the non-finite count that comes with it — in eager, captured and replayed form."""

import numpy as np
import pytest

import oracle
from see_ai_b200 import plan as P
from see_ai_b200 import synth
from see_ai_b200.engine import Engine

pytestmark = pytest.mark.gpu


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


@pytest.mark.parametrize("dims,rank", [((64, 260, 36), 4), ((33, 100, 8), 8), ((31, 516, 300), 16), ((16,) * 100, 12)],
                         ids=["r4", "r8-odd-rows", "r16-wide", "r12-two-tables"])
def test_deltas_are_the_instructions_bits_and_counted(dims, rank):
    blob = synth.build_mlp_plan(synth.MlpConfig(dims=dims, batch=4, rank=rank))
    plan = P.Plan(blob)
    rng = np.random.default_rng(sum(dims))
    arena = plan.stage_arena()
    state = rng.standard_normal(plan.header["persistent_size"] // 4).astype(np.float32)
    arena[:state.nbytes] = state.view(np.uint8)
    ref = oracle.OracleExecutor()
    ref.bind(arena, np.frombuffer(plan.rodata, dtype=np.uint8).copy())
    ref.run(plan.merge)
    eng = Engine(0)
    eng.load(blob)
    eng.set_use_graphs(True)
    eng.write_arena(0, state)
    c0 = eng.backend.counters()
    for _ in range(4):   # eager, captured, replayed
        assert eng.run_merge() is True
        for e in plan.emit:
            assert np.array_equal(eng.read_arena(e.arena_offset, e.byte_size), arena[e.arena_offset:e.arena_offset + e.byte_size])
    assert eng.backend.counters().fused_dispatches > c0.fused_dispatches
    bad = state.copy()
    bad[plan.merge[1].ins[0] // 4] = np.inf   # one row of the first delta
    eng.write_arena(0, bad)
    assert eng.run_merge() is False
    eng.write_arena(0, state)
    assert eng.run_merge() is True
    eng.close()
