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


@pytest.mark.parametrize("graphs", [False, True], ids=["eager", "graphs"])
def test_a_later_write_over_a_delta_is_in_the_finiteness_scan(graphs):
    """An instruction behind the accumulation doubles one delta: finite as accumulated, infinite as it leaves."""
    plan = P.Plan(synth.build_mlp_plan(synth.MlpConfig(dims=(64, 260, 36), batch=4, rank=4)))
    acc = next(i for i in plan.merge if i.opcode == P.Op.GEMM_ACC_NN)
    delta, n = acc.ins[2], acc.out[0] * acc.out[1]
    merge = list(plan.merge) + [P.Instr(P.Op.ADD_EW, 0, 0, (delta, delta, delta, P.NULL_REF), (n, 0, 0))]
    persist = plan.persist_init
    blob = P.write_plan(plan.header, plan.train, plan.eval, merge, plan.step, plan.rodata, persist, emit=plan.emit)
    eng = Engine(0)
    eng.load(blob)
    eng.set_use_graphs(graphs)
    state = np.zeros(plan.header["persistent_size"] // 4, np.float32)
    M, N, K = acc.out
    state[acc.ins[0] // 4:acc.ins[0] // 4 + M * K] = 1.0
    b = state[acc.ins[1] // 4:acc.ins[1] // 4 + K * N]
    for value, finite in ((1.0, True), (6e37, False), (1.0, True)):   # K = 4 terms: 2.4e38 times alpha, then twice that
        b[:] = value / np.frombuffer(np.uint32(acc.ins[3] & 0xFFFFFFFF).tobytes(), np.float32)[0]
        eng.write_arena(0, state)
        for _ in range(3):
            assert eng.run_merge() is finite
            assert np.isfinite(eng.read_arena(delta, 4 * n).view(np.float32)).all() == finite
    eng.close()
