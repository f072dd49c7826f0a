"""Softmax cross-entropy of wide rows: the three launch shapes (256, 512 and 1024 threads to a row) at the edges of
their ranges, more rows than blocks, labels at the row's ends and masked ones, against double precision; and the evaluation tail's chain and tally over more rows than one of
its chunks holds."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from see_ai_b200.engine import Engine
from tests import runloop as R
from tests.test_gpu_engine_tails import _tail_plan
from tests.test_oracle_pinned import Arena

import oracle

pytestmark = pytest.mark.gpu
Op = P.Op


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


@pytest.mark.parametrize("masked", [False, True], ids=["plain", "masked"])
@pytest.mark.parametrize("rows,classes", [(1, 4096), (700, 4100), (3, 8192), (5, 8196), (310, 16384), (2, 16388), (151, 32000),
                                          (7, 32764), (4, 32768)])
def test_wide_rows_against_double(rows, classes, masked):
    rng = np.random.default_rng(rows + classes)
    a = Arena(rng)
    logits = a.alloc(rows * classes, "normal")
    labels = a.alloc(rows)
    loss, probs = a.alloc(1), a.alloc(rows * classes)
    arena, ro = a.build()
    x = arena[logits:logits + 4 * rows * classes].view(np.float32).reshape(rows, classes)
    x *= np.float32(4.0)
    y = rng.integers(0, classes, size=rows, dtype=np.int32)
    y[0] = classes - 1
    if rows > 1:
        y[1] = 0
    if masked and rows > 1:
        y[rows // 2] = -1
    arena[labels:labels + 4 * rows] = y.view(np.uint8)
    be = B.CudaBackend(0)
    be.bind(arena, ro)
    be.run([P.Instr(Op.XENT_MASKED_FWD if masked else Op.XENT_FWD, 0, 0, (logits, labels, loss, probs), (rows, classes, 0))])
    be.close()
    z = x.astype(np.float64)
    p = np.exp(z - z.max(axis=1, keepdims=True))
    p /= p.sum(axis=1, keepdims=True)
    got = arena[probs:probs + 4 * rows * classes].view(np.float32).reshape(rows, classes)
    # the hardware exponential (2^-22 relative), its argument rounded at |x - max| up to 40 or so, f32 sums of 32 terms
    assert np.max(np.abs(got - p) / p) < 1e-5
    live = y >= 0
    want = -np.log(np.maximum(p[np.arange(rows)[live], y[live]], 1e-12)).mean()
    assert abs(float(arena[loss:loss + 4].view(np.float32)[0]) - want) <= 1e-5 * abs(want)


@pytest.mark.parametrize("rows,classes", [(1, 4096), (600, 5000), (700, 8000), (3, 8192), (300, 8196), (5, 16384)])
def test_the_bits_do_not_depend_on_the_threads_to_a_row(rows, classes):
    """A row padded with -inf to 32768 columns (1024 threads to a row) has the same sums, with zeros added."""
    rng = np.random.default_rng(rows + classes)
    x = (rng.standard_normal((rows, classes)) * 4.0).astype(np.float32)
    y = rng.integers(0, classes, size=rows, dtype=np.int32)

    def run(width):
        a = Arena(rng)
        logits = a.alloc(rows * width, np.pad(x, ((0, 0), (0, width - classes)), constant_values=-np.inf))
        labels = a.alloc(rows, y.view(np.float32))
        loss, probs = a.alloc(1), a.alloc(rows * width)
        arena, ro = a.build()
        be = B.CudaBackend(0)
        be.bind(arena, ro)
        be.run([P.Instr(Op.XENT_FWD, 0, 0, (logits, labels, loss, probs), (rows, width, 0))])
        be.close()
        return (arena[probs:probs + 4 * rows * width].view(np.float32).reshape(rows, width)[:, :classes].copy(),
                arena[loss:loss + 4].view(np.float32)[0])

    (p, l), (q, m) = run(classes), run(32768)
    assert np.array_equal(p, q) and l == m


@pytest.mark.parametrize("rows,classes", [(223, 128), (224, 132), (225, 1024), (700, 131)])
def test_eval_tail_over_several_chunks_of_rows(rows, classes):
    rng = np.random.default_rng(rows)
    probs = rng.random((rows, classes)).astype(np.float32)
    probs /= probs.sum(axis=1, keepdims=True)
    labels = np.where(rng.random(rows) < 0.5, probs.argmax(axis=1), rng.integers(0, classes, size=rows)).astype(np.int32)
    probs[3, :] = 0.001; probs[3, 4] = 0.4; probs[3, classes - 1] = 0.4; labels[3] = 4   # the first of two maxima wins
    labels[5::17] = -1
    blob = _tail_plan(rows, classes, True)
    eng = Engine(0)
    eng.load(blob)
    gpu, cpu = R.GpuStepper(eng), R.CpuStepper(P.Plan(blob), oracle.OracleExecutor())
    for real in (rows, rows - 1, 1):
        eg, ec = gpu.evaluate(probs.reshape(-1), labels, real), cpu.evaluate(probs.reshape(-1), labels, real)
        assert (eg.rows, eg.correct, eg.loss_rows) == (ec.rows, ec.correct, ec.loss_rows)
        assert abs(eg.real_row_loss - ec.real_row_loss) <= 1e-12 * max(1.0, abs(ec.real_row_loss))
    eng.close()
