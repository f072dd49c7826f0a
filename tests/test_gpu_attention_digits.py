"""Exact attention by digits, forced wherever it takes the geometry and counted: every form at the edges of 128 queries and 64
keys against float64, score by score too, and no further from it than the strict seam's f32 sums, also where features and
elements differ widely in size; rows without digits against the strict seam; and which of two kernels is taken unasked."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_gpu_attention_exact import _program
from tests.test_gpu_attention_slices import OPS, _float64, _outputs
from tests.util import compare

pytestmark = pytest.mark.gpu
Op = P.Op

# B, S, H, d, and how many of the three instructions take the kernel unasked (a device of 148 SMs).
SHAPES = [
    (24, 127, 4, 64, 1), (24, 128, 4, 64, 3), (8, 300, 12, 64, 3), (10, 321, 10, 60, 1), (32, 64, 8, 64, 1), (16, 64, 4, 64, 0),
    (12, 129, 8, 64, 0), (24, 128, 4, 20, 1), (26, 101, 4, 4, 1), (24, 193, 4, 32, 1),
    (1, 1, 1, 64, 0), (2, 63, 2, 4, 0), (3, 65, 3, 20, 0), (1, 257, 2, 64, 1),
]


def _run(prog, arena, lazy, use=1):
    out = arena.copy()
    be = B.CudaBackend(0)
    if lazy:
        be.set_coherence(B.COHERENCE_LAZY)
        be.set_attention_slices(use)
    be.bind(out, None)
    be.set_program(prog)
    be.run(None)
    be.host_needs(0, out.size)
    be.flush()
    count = be.attention_slices()
    be.close()
    return out, count


def _three(shape, use=2):
    """The three instructions of a geometry, inputs, and a function that runs them: all by the kernel, or by the strict seam."""
    prog, arena = _program(*shape, 0, cached=True)
    prog = [i for i in prog if i.opcode in OPS]

    def run(lazy):
        out, count = _run(prog, arena, lazy, use)
        assert count == (len(OPS) if lazy and use == 2 else 0 if not lazy else count)
        return _outputs(prog, out, *shape)

    return prog, arena, run


def _check(got, strict, want, S, same=1.03, most=np.inf):
    for name, w in want.items():
        err = np.linalg.norm(got[name] - w) / np.linalg.norm(w)
        before = np.linalg.norm(strict[name] - w) / np.linalg.norm(w)
        # A rounding to f32 is 2.5e-8 rms of the value; scores and probabilities carry one or two, sums of up to 321 f32
        # products more.  What the digits leave out is at most 2^-29 of a row's largest score, i.e. nothing that 3 % would not hold.
        # (1e-12: geometries of a few elements that the strict seam has exactly.)
        assert err <= same * before + 1e-12 and before < most, (name, err, before)
    # Score by score: a rounding (2^-24 of it), and 128 products of a residue, uniform within 2^-33 of its row's 2^e, with an element: six
    # standard deviations of their sum are 39 x 2^-33 of 2^(eq + ek), which is at most 2^4 of the row's largest score: 2^-23.7 of that.
    w, g = want["dP"].reshape(-1, S), got["dP"].reshape(-1, S)
    assert (np.abs(g - w) <= 2.0 ** -24 * np.abs(w) + 2.0 ** -23.7 * np.abs(w).max(-1, keepdims=True)).all()
    upper = ~np.tril(np.ones((S, S), dtype=bool))
    for name in ("P", "dP"):
        assert not got[name].reshape(-1, S, S)[:, upper].any(), name


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s[:4])) for s in SHAPES])
def test_against_float64(shape):
    shape = shape[:4]
    prog, arena, run = _three(shape)
    # (Of a geometry of few rows one rounding that falls the other way is more than 3 %.)
    _check(run(True), run(False), _float64(prog, arena, *shape), shape[1], 1.03 if shape[0] * shape[1] * shape[2] > 1000 else 1.3, 3e-7)


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s[:4])) for s in SHAPES])
def test_what_takes_the_kernel_unasked(shape):
    prog, arena = _program(*shape[:4], 0, cached=True)
    prog = [i for i in prog if i.opcode in OPS]
    assert _run(prog, arena, True)[1] == shape[4]
    assert _run(prog, arena, True, use=0)[1] == 0


def _spread(x, what, rng):
    """Features and elements of different sizes, in Q against K and in dO against V."""
    d = x["q"].shape[-1]
    if what.startswith("gains"):
        gain = np.exp2(rng.uniform(-1, 1, size=(x["q"].shape[2], d)) * float(what[5:])).astype(np.float32)
    for a, b in (("q", "k"), ("do", "v")):
        if what.startswith("gains"):             # an ordinary reparametrisation
            x[a] *= gain
            x[b] /= gain
        elif what.startswith("feature"):         # one outlier
            x[a][..., 3] *= np.float32(what[7:])
            x[b][..., 3] /= np.float32(what[7:])
        elif what == "unmet":                    # a large element that meets none, in every row
            x[a][..., 0], x[b][..., 0] = 2.0 ** 34, 0.0
            x[a][..., 1:], x[b][..., 1:] = 1.0, 1.0
        elif what == "unmet_rows":               # ... in some rows
            x[a][:, ::7, :, 0] = 2.0 ** 34
            x[b][..., 0] = 0.0
        elif what == "within_rows":
            x[a] *= np.exp2(rng.uniform(-12, 12, size=x[a].shape)).astype(np.float32)
            x[b] *= np.exp2(rng.uniform(-12, 12, size=x[b].shape)).astype(np.float32)
        elif what == "orthogonal":               # to a mean of the keys a hundred times as large as what they differ by
            m = 100.0 * rng.standard_normal(d)
            x[b] += m.astype(np.float32)
            x[a] -= np.outer(x[a].reshape(-1, d).astype(np.float64) @ m, m / (m @ m)).reshape(x[a].shape).astype(np.float32)
        elif what == "small":                    # gradients, some rows far smaller than others
            x[a] *= np.exp2(rng.uniform(-85, -20, size=x[a].shape[:3]))[..., None].astype(np.float32)


@pytest.mark.parametrize("what", ["gains2", "gains4", "gains8", "gains12", "gains20", "feature1e3", "feature1e4", "feature1e5",
                                  "feature1e6", "unmet", "unmet_rows", "within_rows", "orthogonal", "small"])
@pytest.mark.parametrize("shape", [(24, 128, 4, 64), (3, 321, 2, 36)], ids=["24x128x4x64", "3x321x2x36"])
def test_sizes_that_differ_within_a_row(shape, what):
    Bq, S, H, d = shape
    prog, arena, run = _three(shape)
    fwd, dp, _ = prog
    x = {n: arena[off:off + 4 * Bq * S * H * d].view(np.float32).reshape(Bq, S, H, d)
         for n, off in zip(("q", "k", "v", "do"), (*fwd.ins[:3], dp.ins[0]))}
    v = x["v"].copy()
    _spread(x, what, np.random.default_rng(7))
    want, strict, got = _float64(prog, arena, *shape), run(False), run(True)
    if what == "small":   # (scores near 0: a probability is their exponential all the same)
        want.pop("stats")
    if np.abs(x["v"]).max() > 1e3 * np.abs(v).max():   # one feature of O is nearly all of its norm
        scale = np.abs(want["o"].reshape(-1, d)).max(0, keepdims=True)
        for r in (want, strict, got):
            for name in ("o", "o2"):
                r[name] = (r[name].reshape(-1, d) / scale).reshape(-1)
    _check(got, strict, want, S)


@pytest.mark.parametrize("shape", [(24, 128, 4, 64), (2, 200, 3, 20)], ids=["24x128x4x64", "2x200x3x20"])
@pytest.mark.parametrize("what", ["inf_q", "nan_k", "minus_inf_k", "inf_v", "nan_v", "huge_q", "tiny_k", "zero_rows", "nan_all", "inf_scores",
                                  "nan_last_tile", "large_v", "large_v_rising"])
def test_rows_without_digits(what, shape):
    Bq, S, H, d = shape
    prog, arena, run = _three(shape)
    fwd, dp, _ = prog
    x = {n: arena[off:off + 4 * Bq * S * H * d].view(np.float32).reshape(Bq, S, H, d)
         for n, off in zip(("q", "k", "v", "do"), (*fwd.ins[:3], dp.ins[0]))}
    if what == "inf_q":
        x["q"][1, 5, 2, 7] = np.inf
    elif what == "nan_k":
        x["k"][1, 77, 1, 3] = np.nan
    elif what == "minus_inf_k":
        x["k"][0, 70, H - 1, 9] = -np.inf
    elif what == "inf_v":
        x["v"][1, 100, 0, d - 1] = np.inf
    elif what == "nan_v":
        x["v"][1, 3, 0, 0] = np.nan
    elif what == "huge_q":
        x["q"][:, 9] *= np.float32(1e25)
        x["k"][:, 4] *= np.float32(1e-25)
        x["do"][:, 9] *= np.float32(1e25)
    elif what == "tiny_k":
        x["k"][:, 64:] *= np.float32(1e-30)
        x["v"][:, ::3] *= np.float32(1e-30)
    elif what == "nan_all":
        for t in x.values():
            t[:] = np.nan
    elif what == "inf_scores":                   # finite rows whose products are not, of both signs
        x["q"][:, S // 2] *= np.float32(1e25)
        x["k"][:, 3] *= np.float32(1e25)
        x["do"][:, S // 2] *= np.float32(1e25)
        x["v"][:, 3] *= np.float32(1e25)
    elif what == "nan_last_tile":                # a whole tile of queries without digits, and the one before it with them
        x["q"][:, 128:] = np.nan
        x["do"][:, 128:] = np.nan
    elif what.startswith("large_v"):             # sums that are not normalised would overflow
        x["q"][:] = np.float32(1.0) / np.float32(d)
        x["k"][:] = (np.arange(S, dtype=np.float32) * np.float32(7.5 / S * np.sqrt(d)))[None, :, None, None] if what.endswith("rising") else 1.0
        x["v"][:] = np.float32(9e35)
    else:
        x["q"][:, 3] = 0.0
        x["k"][:, 0:40] = 0.0
        x["do"][1] = 0.0
    with np.errstate(all="ignore"):
        got, want = run(True), run(False)
        for name, w in want.items():
            ok, ratio = compare(np.ascontiguousarray(got[name]).tobytes(), np.ascontiguousarray(w).tobytes(), 1e-5, 1e-7)
            assert ok, (name, ratio)


def test_the_same_sequence_on_both_sides_of_the_rule():
    """Batches just below and above where the kernel becomes the shorter way give a sequence the same results up to rounding."""
    S, H, d = 128, 4, 64
    sides = {}
    for Bq in range(2, 25):
        prog, arena = _program(Bq, S, H, d, 0, cached=True)
        prog = [i for i in prog if i.opcode == Op.ATTN_FWD_TILED]
        n = S * H * d
        refs = (*prog[0].ins[:3],)
        rng = np.random.default_rng(3)
        for off in refs:   # the same first sequence, with outlier features that cancel
            seq = rng.standard_normal((S, H, d), dtype=np.float32)
            if off != refs[2]:
                seq[..., 5] *= np.float32(1e4 if off == refs[0] else 1e-4)
            arena[off:off + 4 * n].view(np.float32)[:] = seq.reshape(-1)
        out, count = _run(prog, arena, True)
        sides[count] = out[prog[0].ins[3]:prog[0].ins[3] + 4 * n].tobytes()
        if len(sides) == 2:
            break
    assert sorted(sides) == [0, 1]
    # (Two f32 sums of up to 128 weighted values, each with its own roundings: 1e-6 of the scale.)
    ok, ratio = compare(sides[1], sides[0], 1e-6, 0.0)
    assert ok, ratio
