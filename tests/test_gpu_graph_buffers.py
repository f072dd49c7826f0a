"""Ranges of one engine that need more scratch than an earlier, captured one: evaluation
is captured, training then replaces the buffers its graph addresses, evaluation follows.
Every pass gives the bits of an engine without graphs."""

import numpy as np
import pytest

from see_ai_b200 import plan as P
from see_ai_b200 import synth
from see_ai_b200.engine import Engine

pytestmark = pytest.mark.gpu

PLANS = {
    "int8-odd-vocabulary": dict(layers=1, d_model=256, heads=4, ffn=1024, vocab=2001, seq=200, batch_seqs=3, rank=8, alpha=16.0,
                                targets=("q", "v"), quantized=True, attention="tiled"),
    "f32": dict(layers=2, d_model=128, heads=4, ffn=512, vocab=1000, seq=64, batch_seqs=4, rank=8, alpha=16.0,
                targets=("q", "v"), quantized=False, attention="cached"),
}


@pytest.mark.parametrize("plan", PLANS, ids=list(PLANS))
def test_evaluate_train_evaluate_under_graphs(plan):
    blob = synth.build_decoder_plan(synth.DecoderConfig(**PLANS[plan]))
    p = P.Plan(blob)
    rows, vocab = p.header["batch"], PLANS[plan]["vocab"]
    grads = [(i.ins[1], 4 * i.out[0]) for i in p.train if i.opcode == P.Op.ADAMW_STEP]
    loss = next(i for i in p.eval if i.opcode == P.Op.XENT_FWD)

    def passes(graphs):
        rng = np.random.default_rng(3)
        eng = Engine(0)
        eng.load(blob)
        eng.set_use_graphs(graphs)
        out = []
        for kind in "EEETTTEETE":
            x = rng.integers(0, vocab, size=rows, dtype=np.int32)
            y = rng.integers(0, vocab, size=rows, dtype=np.int32)
            if kind == "E":
                r = eng.evaluate_rows(x, y, rows)
                out.append([np.float32(r.loss).tobytes(), r.correct, eng.read_arena(loss.ins[3], 4 * rows * vocab).tobytes()])
            else:
                out.append([np.float32(eng.train_step(x, y)).tobytes()] + [eng.read_arena(o, n).tobytes() for o, n in grads])
        out.append([eng.read_arena(0, p.header["persistent_size"]).tobytes()])
        assert eng.backend.counters().split_executions > 0
        eng.close()
        return out

    for i, (a, b) in enumerate(zip(passes(True), passes(False))):
        assert a == b, f"pass {i}"
