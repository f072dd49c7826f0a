"""The relaxed tiled forward of sequences of several query tiles (two tiles of a (sequence, head) at a time on a
persistent CTA) against float64, where a CTA walks several pairs: an odd number of tiles, tiles that end inside a step,
both head widths, scores whose maximum moves late (the output is rescaled)."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_gpu_umma import bf16_round
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op


def _forward(x, Bq, S, H, d):
    a = Arena(np.random.default_rng(0))
    refs = [a.alloc(x[n].size, x[n]) for n in ("q", "k", "v")]
    o, stats = a.alloc(x["q"].size), a.alloc(Bq * H * S * 4)
    arena, ro = a.build()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.bind(arena, ro)
    be.run([P.Instr(Op.ATTN_FWD_TILED, P.FLAG_RELAXED, 0, (*refs, o), (stats, P.pack2(Bq, S), P.pack2(H, d)))])
    assert be.counters().relaxed_executions == 1
    be.host_needs(0, arena.size)
    be.flush()
    be.close()
    n = Bq * H * S
    return (arena[o:o + 4 * x["q"].size].view(np.float32).reshape(Bq, S, H, d).copy(),
            arena[stats:stats + 16 * n].view(np.float32).reshape(Bq, H, S, 4).copy())


def _inputs(rng, Bq, S, H, d):
    x = {n: bf16_round(rng.standard_normal(Bq * S * H * d).astype(np.float32)).reshape(Bq, S, H, d) for n in ("q", "k", "v")}
    x["k"] = bf16_round((x["k"] * (1.0 + 2.0 * np.arange(S) / S)[None, :, None, None]).astype(np.float32).reshape(-1)).reshape(x["k"].shape)
    return x


# 3 rounds of a CTA's pairs and an odd number of tiles; one pair a sequence; two rounds at d = 128 (one output buffer);
# a last tile of one step, of two.
GEOMS = [(8, 520, 20, 64), (56, 136, 12, 64), (9, 264, 20, 128), (20, 200, 16, 128), (2, 1160, 40, 64)]


@pytest.mark.parametrize("geom", GEOMS, ids=["B%dS%dH%dd%d" % g for g in GEOMS])
def test_several_pairs_to_a_cta_against_float64(geom):
    import torch
    Bq, S, H, d = geom
    x = _inputs(np.random.default_rng(S + d + H), *geom)
    o, stats = _forward({n: v.reshape(-1) for n, v in x.items()}, *geom)
    above = torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1)
    for b in range(Bq):
        q, k, v = (torch.from_numpy(x[n][b]).cuda().double().transpose(0, 1) for n in ("q", "k", "v"))   # [H, S, d]
        s = (q @ k.transpose(1, 2) / d ** 0.5).masked_fill(above, float("-inf"))
        p = torch.softmax(s, dim=-1)
        want, mag = (p @ v).transpose(0, 1).cpu().numpy(), (p @ v.abs()).transpose(0, 1).cpu().numpy()
        # P rounds to bf16 once: eight significant bits, so at most 2^-8 of each p.  Scores of up to 60, truncated at
        # 2^-22 of themselves or so, are exponents.
        worst = float((np.abs(o[b] - want) / (mag + 1e-7)).max())
        assert worst <= 2.0 ** -8 + 1e-4, (b, worst)
        m = s.max(dim=-1).values
        inv = 1.0 / torch.exp(s - m[..., None]).sum(dim=-1)
        assert np.abs(stats[b, :, :, 0] - m.cpu().numpy()).max() <= 1e-4
        assert np.abs(stats[b, :, :, 1] / inv.cpu().numpy() - 1.0).max() <= 2e-4


@pytest.mark.parametrize("geom", [(32, 136, 12, 64), (3, 520, 8, 64), (5, 264, 6, 128)], ids=lambda g: "B%dS%dH%dd%d" % g)
def test_the_first_tile_has_the_bits_of_a_sequence_that_is_only_that(geom):
    """Causal: the first 128 positions know nothing of the rest, and a sequence of 128 has the one-tile kernel."""
    Bq, S, H, d = geom
    x = _inputs(np.random.default_rng(S + d), *geom)
    o, stats = _forward({n: v.reshape(-1) for n, v in x.items()}, *geom)
    one, one_stats = _forward({n: np.ascontiguousarray(v[:, :128]).reshape(-1) for n, v in x.items()}, Bq, 128, H, d)
    assert np.array_equal(o[:, :128], one)
    assert np.array_equal(stats[:, :, :128], one_stats)


# (batches of the same sequences, S, H, d): either side of each line between the two kernels.
LINES = [((2, 26), 192, 12, 64), ((16, 22), 256, 12, 64), ((8, 12, 16, 22), 320, 12, 64), ((4, 22), 136, 8, 128), ((2, 22), 256, 8, 128)]


@pytest.mark.parametrize("line", LINES, ids=lambda l: "S%dH%dd%d" % l[1:])
def test_a_sequence_has_the_same_bits_in_every_batch(line):
    batches, S, H, d = line
    x = _inputs(np.random.default_rng(S + d), max(batches), S, H, d)
    o, stats = _forward({n: v.reshape(-1) for n, v in x.items()}, max(batches), S, H, d)
    for b in batches[:-1]:
        few, few_stats = _forward({n: np.ascontiguousarray(v[:b]).reshape(-1) for n, v in x.items()}, b, S, H, d)
        assert np.array_equal(few, o[:b]) and np.array_equal(few_stats, stats[:b])
