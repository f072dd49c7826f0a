"""Input gradients that several relaxed products add up to, launched together (a chain), alone and where something else
that is launched together lies between the members: a second chain, or Q, K and V side by side.  A program run as ONE
range is compared with the same program run one instruction per range: the frozen products are the same bf16 computation
both ways, so the sums differ by the arithmetic of the low-rank terms and of the additions, held to 2e-6 of the terms'
magnitudes as the folds are.  And with the same range whose products are launched one by one: the same bits."""

import numpy as np
import pytest

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.test_oracle_pinned import Arena

pytestmark = pytest.mark.gpu
Op = P.Op
REL, CS, ADDEND = P.FLAG_RELAXED, P.FLAG_Q8_COL_SCALE, P.FLAG_GEMM_ADDEND
SIZES = [(256, 128, 192), (4864, 128, 2048)]   # (M, K, N): one-tile kernel; persistent kernel


class Chain:
    """s_p = s_(p-1) + dT_p A_p^T + dY_p W_p^T, p = 0 .. n - 1: the instructions of each member, and what is scratch."""

    def __init__(self, a, rng, M, N, K, r, n):
        self.M, self.N, self.K, self.r = M, N, K, r
        self.members, self.scratch, self.terms = [], [], []
        total = None
        for p in range(n):
            dy, dt, A = a.alloc(M * K, "normal"), a.alloc(M * r, "normal"), a.alloc(N * r, "normal", scale=0.05)
            levels = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
            scale = (rng.random(K) * 0.01 + 1e-3).astype(np.float32)
            w, sk = a.ro_alloc(levels), a.ro_alloc(scale)
            z, part, out = a.alloc(M * N), a.alloc(M * N), a.alloc(M * N)
            g = P.Instr(Op.GEMM_NT_Q8, REL | CS, 0, (dy, w, z, sk), (M, N, K))
            if p == 0:
                self.members.append([g, P.Instr(Op.GEMM_NT, ADDEND, 0, (dt, A, out, z), (M, N, r))])
            else:
                self.members.append([P.Instr(Op.GEMM_NT, ADDEND, 0, (dt, A, part, total), (M, N, r)), g,
                                     P.Instr(Op.ADD_EW, 0, 0, (part, z, out, P.NULL_REF), (M * N, 0, 0))])
                self.scratch.append(part)
                self.scratch.append(total)
            self.scratch.append(z)
            self.terms.append((dy, levels * scale, dt, A))
            total = out
        self.out = total

    def fills(self):
        return [P.Instr(Op.FILL, 0, 0, (s, P.f32_bits(0.0)), (self.M * self.N, 0, 0)) for s in self.scratch]

    def check(self, one, split, arena0):
        M, N, K, r = self.M, self.N, self.K, self.r
        got, want = _f32(one, self.out, M * N), _f32(split, self.out, M * N)
        mag = np.ones((M, N))
        for dy, w, dt, A in self.terms:
            mag += np.abs(_f32(arena0, dy, M * K).reshape(M, K) @ w.T)
            mag += np.abs(_f32(arena0, dt, M * r).reshape(M, r)) @ np.abs(_f32(arena0, A, N * r).reshape(N, r)).T
        mag = mag.reshape(-1)
        err = np.abs(got - want) / mag
        assert np.isfinite(got).all() and err.max() < 2e-6, err.max()


def _f32(arena, off, n):
    return arena[off:off + 4 * n].view(np.float32).astype(np.float64)


def _run(prog, arena0, ro, one_range=True, groups=True):
    arena = arena0.copy()
    be = B.CudaBackend(0)
    be.set_coherence(B.COHERENCE_LAZY)
    be.set_product_groups(groups)
    be.bind(arena, ro)
    be.set_program(prog)
    for i, end in [(0, len(prog))] if one_range else [(i, i + 1) for i in range(len(prog))]:
        be.run(None, None, i, end)
    be.host_needs(0, arena.size)
    be.flush()
    launches = be.counters().kernel_launches
    be.close()
    return arena, launches


@pytest.mark.parametrize("size", SIZES, ids=["one-tile", "persistent"])
@pytest.mark.parametrize("n", [2, 3])
def test_two_interleaved_chains(size, n):
    M, K, N = size
    rng = np.random.default_rng(M + n)
    a = Arena(rng)
    one, two = (Chain(a, rng, M, N, K, 16, n) for _ in range(2))
    prog = [ins for p in range(n) for c in (one, two) for ins in c.members[p]] + one.fills() + two.fills()
    arena0, ro = a.build()
    got, _ = _run(prog, arena0, ro)
    want, _ = _run(prog, arena0, ro, one_range=False)
    one.check(got, want, arena0)
    two.check(got, want, arena0)


@pytest.mark.parametrize("M", [256, 4864])
def test_side_by_side_products_inside_a_chain(M):
    S, H, d, K, r = 64, 2, 64, 128, 16
    N = H * d
    rng = np.random.default_rng(M)
    a = Arena(rng)
    chain = Chain(a, rng, M, N, K, r, 2)
    x = a.alloc(M * K, "normal")
    q, k, v, o = (a.alloc(M * N) for _ in range(4))
    stats = a.alloc(M * H * 4)
    qkv = [P.Instr(Op.GEMM_NN_Q8, REL | CS, 0,
                   (x, a.ro_alloc(rng.integers(-127, 128, size=K * N, dtype=np.int8)), out,
                    a.ro_alloc((rng.random(N) * 0.001 + 1e-3).astype(np.float32))), (M, N, K)) for out in (q, k, v)]
    attention = P.Instr(Op.ATTN_FWD_TILED, REL, 0, (q, k, v, o), (stats, P.pack2(M // S, S), P.pack2(H, d)))
    clear = [P.Instr(Op.FILL, 0, 0, (t, P.f32_bits(0.0)), (M * N, 0, 0)) for t in (q, k, v)]
    prog = chain.members[0] + qkv + [attention] + clear + chain.members[1] + chain.fills()
    arena0, ro = a.build()
    got, _ = _run(prog, arena0, ro)
    want, _ = _run(prog, arena0, ro, one_range=False)
    chain.check(got, want, arena0)
    assert np.array_equal(got[o:o + 4 * M * N], want[o:o + 4 * M * N])


# (M, N, K, rank, members): the one-tile kernel at each width and cut, the persistent one, CTA pairs; ragged
# last tiles in both directions; one and two low-rank blocks.
CHAINS = [
    (64, 64, 64, 4, 2), (200, 128, 128, 16, 3), (600, 512, 512, 8, 3), (600, 768, 768, 16, 3), (300, 768, 768, 8, 2),
    (1000, 516, 520, 16, 3), (2000, 256, 256, 16, 3), (4096, 768, 768, 16, 3), (4001, 768, 768, 16, 2),
    (4864, 2048, 192, 16, 3), (20000, 768, 320, 8, 3), (20000, 1028, 768, 16, 2),
]


@pytest.mark.parametrize("shape", CHAINS, ids=["x".join(map(str, c)) for c in CHAINS])
def test_a_chain_has_the_separate_launches_bits(shape):
    M, N, K, r, n = shape
    rng = np.random.default_rng(M + N + K)
    a = Arena(rng)
    chain = Chain(a, rng, M, N, K, r, n)
    prog = [ins for m in chain.members for ins in m] + chain.fills()
    arena0, ro = a.build()
    got, launches = _run(prog, arena0, ro)
    want, launches_one_by_one = _run(prog, arena0, ro, groups=False)
    assert np.array_equal(got[chain.out:chain.out + 4 * M * N], want[chain.out:chain.out + 4 * M * N])
    assert np.isfinite(_f32(got, chain.out, M * N)).all()
    assert launches_one_by_one - launches in (0, n - 1)   # (0: the planner found one by one the shorter)
    if M >= 4000:
        assert launches_one_by_one - launches == n - 1


# The one-tile kernel with and without a cut, the persistent one, CTA pairs; rows that end inside a tile.
QKV = [(192, 64, 128, 128), (600, 200, 512, 512), (600, 200, 768, 768), (304, 304, 768, 768), (512, 128, 768, 768),
       (4096, 512, 768, 768), (20000, 160, 256, 192)]


@pytest.mark.parametrize("shape", QKV, ids=["x".join(map(str, c)) for c in QKV])
@pytest.mark.parametrize("n", [2, 3])
def test_products_side_by_side_have_the_separate_launches_bits(shape, n):
    M, S, N, K = shape
    d, H = 64, N // 64
    rng = np.random.default_rng(M + N + K + n)
    a = Arena(rng)
    x = a.alloc(M * K, "normal")
    q, k, v, o = (a.alloc(M * N, "normal") for _ in range(4))
    stats = a.alloc(M * H * 4)
    outs = (q, k, v)[:n]
    products = [P.Instr(Op.GEMM_NN_Q8, REL | CS, 0,
                        (x, a.ro_alloc(rng.integers(-127, 128, size=K * N, dtype=np.int8)), out,
                         a.ro_alloc((rng.random(N) * 0.001 + 1e-3).astype(np.float32))), (M, N, K)) for out in outs]
    attention = P.Instr(Op.ATTN_FWD_TILED, REL, 0, (q, k, v, o), (stats, P.pack2(M // S, S), P.pack2(H, d)))
    clear = [P.Instr(Op.FILL, 0, 0, (t, P.f32_bits(0.0)), (M * N, 0, 0)) for t in outs]
    prog = products + [attention] + clear
    arena0, ro = a.build()
    got, launches = _run(prog, arena0, ro)
    want, launches_one_by_one = _run(prog, arena0, ro, groups=False)
    assert np.array_equal(got[o:o + 4 * M * N], want[o:o + 4 * M * N])
    assert np.array_equal(got[stats:stats + 16 * M * H], want[stats:stats + 16 * M * H])
    assert launches_one_by_one - launches in (0, n - 1)
    if M >= 4000:
        assert launches_one_by_one - launches == n - 1
