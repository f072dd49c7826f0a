"""The exact attention family on the tensor cores (lazy coherence, geometries with enough whole tiles): scores from
fixed-point digits, output sums from bf16 pieces.  Edges of 128 queries and 64 keys, heads of 4 to 64 features, one walk over
the keys (statistics) and two (probabilities), raw scores; against float64, and no further from it than the f32 sums of the
strict seam; and rows that have no digits, against the strict seam."""

import numpy as np
import pytest
import torch

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_gpu_attention_exact import _program
from tests.util import compare

pytestmark = pytest.mark.gpu
Op = P.Op
OPS = (Op.ATTN_FWD, Op.ATTN_DP, Op.ATTN_FWD_TILED)

SHAPES = [   # B, S, H, d: all three instructions are the kernel's
    (32, 64, 8, 64), (24, 127, 4, 64), (24, 128, 4, 64), (8, 300, 12, 64), (10, 321, 10, 60),
]
ONE_WALK = [   # the statistics form, and of the narrow heads the probabilities
    (16, 64, 4, 64), (12, 129, 8, 64), (24, 128, 4, 20), (26, 101, 4, 4), (24, 193, 4, 32),
]


def _run(prog, arena, lazy):
    out = arena.copy()
    be = B.CudaBackend(0)
    if lazy:
        be.set_coherence(B.COHERENCE_LAZY)
    be.bind(out, None)
    be.set_program(prog)
    be.run(None)
    be.host_needs(0, out.size)
    be.flush()
    be.close()
    return out


def _outputs(prog, arena, Bq, S, H, d):
    f = lambda off, n: arena[off:off + 4 * n].view(np.float32)
    td, ss = Bq * S * H * d, Bq * H * S * S
    fwd, dp, tiled = prog
    return dict(o=f(fwd.ins[3], td), P=f(fwd.out[0], ss), dP=f(dp.ins[2], ss), o2=f(tiled.ins[3], td),
                stats=f(tiled.out[0], 4 * Bq * H * S).reshape(-1, 4))


def _float64(prog, arena, Bq, S, H, d):
    fwd, dp, _ = prog
    q, k, v, do = (torch.from_numpy(arena[off:off + 4 * Bq * S * H * d].view(np.float32).copy()).cuda().double()
                   .view(Bq, S, H, d).permute(0, 2, 1, 3) for off in (*fwd.ins[:3], dp.ins[0]))
    mask = torch.tril(torch.ones(S, S, device="cuda", dtype=torch.bool))
    s = (q @ k.transpose(-1, -2) / np.sqrt(d)).masked_fill(~mask, -np.inf)
    p = torch.softmax(s, -1)
    o = (p @ v).permute(0, 2, 1, 3).reshape(-1)
    top = s.max(-1).values
    inv = 1.0 / torch.exp(s - top[..., None]).sum(-1)
    stats = torch.stack([top.reshape(-1), inv.reshape(-1), torch.zeros_like(inv).reshape(-1), torch.zeros_like(inv).reshape(-1)], 1)
    dpm = (do @ v.transpose(-1, -2)).masked_fill(~mask, 0.0)
    want = dict(o=o, P=p.reshape(-1), dP=dpm.reshape(-1), o2=o, stats=stats)
    return {name: t.cpu().numpy() for name, t in want.items()}


@pytest.mark.parametrize("shape", SHAPES + ONE_WALK, ids=["x".join(map(str, s)) for s in SHAPES + ONE_WALK])
def test_against_float64(shape):
    prog, arena = _program(*shape, 0, cached=True)
    prog = [i for i in prog if i.opcode in OPS]
    got = _outputs(prog, _run(prog, arena, True), *shape)
    strict = _outputs(prog, _run(prog, arena, False), *shape)
    want = _float64(prog, arena, *shape)
    for name, w in want.items():
        err = np.linalg.norm(got[name] - w) / np.linalg.norm(w)
        before = np.linalg.norm(strict[name] - w) / np.linalg.norm(w)
        # A rounding to f32 is 2.5e-8 rms of the value; scores and probabilities carry one or two, sums of up to 321 f32
        # products more.  The kernel adds 5e-10 to the scores (digits left out), i.e. nothing that 3 % would not hold.
        assert err <= 1.03 * before and before < 3e-7, (name, err, before)
    S = shape[1]
    upper = ~np.tril(np.ones((S, S), dtype=bool))
    for name in ("P", "dP"):
        assert not got[name].reshape(-1, S, S)[:, upper].any(), name


@pytest.mark.parametrize("what", ["inf_q", "nan_k", "minus_inf_k", "inf_v", "nan_v", "huge_q", "tiny_k", "zero_rows"])
def test_rows_without_digits(what):
    Bq, S, H, d = shape = (24, 128, 4, 64)
    prog, arena = _program(*shape, 0, cached=True)
    prog = [i for i in prog if i.opcode in OPS]
    fwd, dp, _ = prog
    x = {n: arena[off:off + 4 * Bq * S * H * d].view(np.float32).reshape(Bq, S, H, d)
         for n, off in zip(("q", "k", "v", "do"), (*fwd.ins[:3], dp.ins[0]))}
    if what == "inf_q":
        x["q"][1, 5, 2, 7] = np.inf
    elif what == "nan_k":
        x["k"][2, 77, 1, 3] = np.nan
    elif what == "minus_inf_k":
        x["k"][0, 70, 3, 9] = -np.inf
    elif what == "inf_v":
        x["v"][3, 100, 0, 63] = np.inf
    elif what == "nan_v":
        x["v"][3, 3, 0, 0] = np.nan
    elif what == "huge_q":
        x["q"][:, 9] *= np.float32(1e25)
        x["k"][:, 4] *= np.float32(1e-25)
        x["do"][:, 9] *= np.float32(1e25)
    elif what == "tiny_k":
        x["k"][:, 64:] *= np.float32(1e-30)
        x["v"][:, ::3] *= np.float32(1e-30)
    else:
        x["q"][:, 3] = 0.0
        x["k"][:, 0:40] = 0.0
        x["do"][1] = 0.0
    with np.errstate(all="ignore"):
        got = _outputs(prog, _run(prog, arena, True), *shape)
        want = _outputs(prog, _run(prog, arena, False), *shape)
        for name, w in want.items():
            ok, ratio = compare(np.ascontiguousarray(got[name]).tobytes(), np.ascontiguousarray(w).tobytes(), 1e-5, 1e-7)
            assert ok, (name, ratio)
