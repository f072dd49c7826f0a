"""Q, K and V's adapter down products in one launch: the bits of one launch each, at the fewest rows, at rows that end inside a
tile, at several tiles to a group of warps, and on both sides of the row count from which they are launched one by one."""

import numpy as np
import pytest

from see_ai_b200 import synth
from tests.test_gpu_product_groups import _steps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("targets,rank", [("qkv", 16), ("qv", 8)])
@pytest.mark.parametrize("seq,seqs", [(64, 1), (72, 3), (512, 8), (512, 37), (512, 38)])
def test_the_bits_of_one_launch_each(seq, seqs, targets, rank):
    cfg = synth.DecoderConfig(layers=1, d_model=768, heads=12, ffn=256, vocab=512, seq=seq, batch_seqs=seqs, rank=rank,
                              alpha=2.0 * rank, targets=tuple(targets), quantized=True, attention="tiled", seed=4)
    got, n_grouped = _steps(cfg, True, 2)
    want, n_single = _steps(cfg, True, 2, groups=False)
    assert n_grouped < n_single
    for (l1, g1), (l2, g2) in zip(got, want):
        assert l1 == l2 and np.array_equal(g1, g2)
