"""What the piece kernels' epilogues absorb, past one round of cut tiles: the one-tile kernel, the persistent one, the one on
CTA pairs, with rows and columns that end inside a tile.  The bits of the separate instructions."""

import numpy as np
import pytest

from tests import test_gpu_exact_epilogues as exact

pytestmark = pytest.mark.gpu

SHAPES = [(2100, 1284, 128), (2100, 3076, 64), (4100, 2308, 128)]


@pytest.mark.parametrize("tail", ["b", "bg", "b+", "bs"])
@pytest.mark.parametrize("kind", ["f32", "q8", "addend"])
@pytest.mark.parametrize("shape", SHAPES, ids=["tile", "persistent", "pairs"])
def test_the_separate_instructions_bits(shape, kind, tail):
    prog, (arena, ro), _ = exact._case(shape, kind, tail)
    got, fused = exact._run(prog, arena, ro, True)
    want, single = exact._run(prog, arena, ro, False)
    np.testing.assert_array_equal(got, want)
    absorbed = len(tail) - (kind == "addend" and "+" in tail)   # (one addend to a product)
    assert fused.fused_dispatches == absorbed == single.kernel_launches - fused.kernel_launches


@pytest.mark.parametrize("tail", ["bs", "bg", "b+"])
@pytest.mark.parametrize("kind", ["f32", "q8"])
@pytest.mark.parametrize("shape", SHAPES + [(2100, 3073, 64)], ids=["tile", "persistent", "pairs", "ragged"])
def test_sums_that_are_not_finite(shape, kind, tail):
    fused, single = exact.sums_that_are_not_finite(shape, kind, tail)
    assert fused.fused_dispatches == len(tail) == single.kernel_launches - fused.kernel_launches
