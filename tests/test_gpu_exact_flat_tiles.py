"""The smallest exact products, whose tiles are 8 x 8: the CPU's bits at the edges of
those tiles, of the 128-wide k slices, and on both sides of the line to 16 x 16."""

import pytest

from tests import test_gpu_exact_flat as flat

pytestmark = pytest.mark.gpu

# 37 and 38 tiles of 16 x 16 are the last count that takes 8 x 8 and the first that does not.
SHAPES = [(8, 8, 128), (7, 9, 127), (9, 7, 129), (1, 25, 300), (15, 8, 255), (16, 37 * 16, 3), (16, 37 * 16 + 1, 3)]


def setup_module(m):
    flat.setup_module(m)


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_bits_of_the_cpu_executor(shape):
    flat.test_bits_of_the_cpu_executor(shape)
