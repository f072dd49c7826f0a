"""Relaxed products launched together (Q, K and V side by side; their input gradients chained into one sum) against the
same step without any fusion, to what bf16 operands leave, and against the same step with every product a launch of its
own, bit for bit: the one-tile kernel, the persistent one and CTA pairs, sites with and
without an adapter, ranks with one and two low-rank blocks; eager, captured and replayed."""

import numpy as np
import pytest

from see_ai_b200 import plan as P
from see_ai_b200 import synth
from see_ai_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _steps(cfg, grouped, steps=1, groups=True):
    blob = synth.build_decoder_plan(cfg)
    plan = P.Plan(blob)
    spans = [(i.ins[1], i.ins[1] + 4 * i.out[0]) for i in plan.train if i.opcode == P.Op.ADAMW_STEP]
    lo, hi = min(s[0] for s in spans), max(s[1] for s in spans)
    rng = np.random.default_rng(9)
    eng = Engine(0)
    eng.backend.set_epilogue_fusion(grouped)   # (off: no group, no fold, every instruction's f32 output stored)
    eng.backend.set_product_groups(groups)
    eng.load(blob)
    eng.set_use_graphs(True)
    state = np.frombuffer(plan.persist_init, dtype=np.uint8).copy().view(np.float32)
    state += rng.standard_normal(state.size).astype(np.float32) * np.float32(0.02)   # B starts at zero: move it
    for i in plan.train:
        if i.opcode == P.Op.ADAMW_STEP:
            for m in (2, 3):
                state[i.ins[m] // 4:i.ins[m] // 4 + i.out[0]] = 0.0
    eng.restore(state.view(np.uint8), 1)
    out = []
    for _ in range(steps):
        rec = rng.integers(0, cfg.vocab, size=(cfg.batch_seqs, cfg.seq + 1), dtype=np.int32)
        loss = eng.train_step(np.ascontiguousarray(rec[:, :-1]).reshape(-1), np.ascontiguousarray(rec[:, 1:]).reshape(-1))
        out.append((loss, eng.read_arena(lo, hi - lo).view(np.float32).astype(np.float64)))
    launches = eng.backend.counters().kernel_launches
    eng.close()
    return out, launches


@pytest.mark.parametrize("targets,rank", [("qkvo", 16), ("qv", 8), ("q", 4), ("k", 8)])
@pytest.mark.parametrize("d_model,seq,seqs", [(128, 72, 3), (512, 512, 40)], ids=["one-tile", "persistent"])
def test_grouped_products_give_the_separate_products_gradients(d_model, seq, seqs, targets, rank):
    cfg = synth.DecoderConfig(layers=2, d_model=d_model, heads=d_model // 64, ffn=256, vocab=512, seq=seq, batch_seqs=seqs,
                              rank=rank, alpha=2.0 * rank, targets=tuple(targets), quantized=True, attention="tiled", seed=3)
    got, n_grouped = _steps(cfg, True, 4)
    want, n_single = _steps(cfg, False, 4)
    assert n_grouped < n_single
    # One step from the same state: the same bf16 operands, sums rounded in other places, and what that turns over in
    # the bf16 copies further on (2^-9 each).
    (l1, g1), (l2, g2) = got[0], want[0]
    assert abs(l1 - l2) <= 1e-4 * abs(l2)
    assert np.isfinite(g1).all() and np.linalg.norm(g1 - g2) <= 1e-2 * np.linalg.norm(g2), np.linalg.norm(g1 - g2) / np.linalg.norm(g2)
    for (l1, _), (l2, _) in zip(got, want):
        assert abs(l1 - l2) <= 1e-3 * abs(l2)


@pytest.mark.parametrize("targets,rank", [("qkvo", 16), ("qv", 8), ("q", 4), ("k", 8), ("qkv", 12)])
@pytest.mark.parametrize("d_model,seq,seqs", [(128, 72, 3), (512, 200, 3), (768, 128, 4), (512, 512, 40)],
                         ids=["one-tile", "ragged", "cut", "persistent"])
def test_grouping_alone_leaves_every_bit(d_model, seq, seqs, targets, rank):
    cfg = synth.DecoderConfig(layers=2, d_model=d_model, heads=d_model // 64, ffn=256, vocab=512, seq=seq, batch_seqs=seqs,
                              rank=rank, alpha=2.0 * rank, targets=tuple(targets), quantized=True, attention="tiled", seed=3)
    got, n_grouped = _steps(cfg, True, 4)
    want, n_single = _steps(cfg, True, 4, groups=False)
    assert n_grouped < n_single or d_model < 512
    for (l1, g1), (l2, g2) in zip(got, want):
        assert l1 == l2 and np.array_equal(g1, g2)
