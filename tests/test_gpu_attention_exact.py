"""The exact attention family at the edges of its kernels' tiles (8, 16 or 32
rows of one axis, 64 of the other, 8 features and 64 output columns at a time,
16-byte and scalar access, rows too long and heads too wide for shared memory), instruction by
instruction from the CPU oracle's bytes: the cached family's products bit for
bit, what holds a double row sum or expf to the 1e-5 of the tensor's scale the
executor is held to everywhere."""

import numpy as np
import pytest

import oracle
from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from tests.util import BIT_EXACT, compare

pytestmark = pytest.mark.gpu
Op = P.Op

SHAPES = [   # B, S, H, d
    (1, 1, 1, 8), (2, 63, 2, 32), (1, 65, 3, 64), (1, 130, 1, 66), (1, 200, 2, 128), (2, 64, 1, 20), (1, 257, 1, 33),
    (10, 70, 10, 12),    # two rows per thread
    (20, 65, 16, 8),     # four
    (1, 700, 1, 16),     # the tiled backward's two score rows: 16-row blocks
    (1, 40, 1, 3400),    # a head too wide for a tile block (the tiled backward of keys stops at 256 features)
    (1, 6900, 1, 8),     # score rows too long for a tile block: one warp per row
]


def setup_module(_m):
    if not oracle.have_oracle():
        oracle.build("oracle")


def _program(Bq, S, H, d, segments, cached, shift=0):
    rng = np.random.default_rng(S * 1000 + d + segments)
    td, ss = Bq * S * H * d, Bq * H * S * S
    refs, size = {}, 0
    sizes = dict(q=td, k=td, v=td, do=td, starts=Bq * S, o=td, dq=td, dk=td, dv=td, o2=td, dq2=td, dk2=td, dv2=td,
                 stats=4 * Bq * H * S)
    if cached:
        sizes.update(P=ss, dP=ss, dS=ss)
    for name, n in sizes.items():
        refs[name] = size + shift
        size = (size + shift + 4 * n + 63) // 64 * 64
    arena = np.zeros(size, dtype=np.uint8)
    for name in ("q", "k", "v", "do"):
        arena[refs[name]:refs[name] + 4 * td] = rng.standard_normal(td, dtype=np.float32).view(np.uint8)
    if segments:   # packed sequences: where each position's own segment begins
        cuts = np.sort(rng.integers(0, S, size=(Bq, 3)), axis=1)
        pos = np.arange(S)
        starts = np.stack([np.max(np.where(c[:, None] <= pos, c[:, None], 0), axis=0) for c in cuts]).astype(np.int32)
        arena[refs["starts"]:refs["starts"] + 4 * Bq * S] = starts.reshape(-1).view(np.uint8)
    o = refs
    bs, hd, geo = P.pack2(Bq, S), P.pack2(H, d), P.pack_attn_geometry(Bq, S, H, d)
    prog = []
    if cached:
        prog += [P.Instr(Op.ATTN_FWD_SEG, 0, 0, (o["q"], o["k"], o["v"], o["o"]), (o["P"], geo, o["starts"])) if segments else
                 P.Instr(Op.ATTN_FWD, 0, 0, (o["q"], o["k"], o["v"], o["o"]), (o["P"], bs, hd)),
                 P.Instr(Op.ATTN_DV, 0, 0, (o["P"], o["do"], o["dv"]), (bs, hd)),
                 P.Instr(Op.ATTN_DP, 0, 0, (o["do"], o["v"], o["dP"]), (bs, hd)),
                 P.Instr(Op.SOFTMAX_ROWS_BWD, 0, 0, (o["P"], o["dP"], o["dS"]), (P.pack2(Bq * H * S, S),)),
                 P.Instr(Op.ATTN_DQ, 0, 0, (o["dS"], o["k"], o["dq"]), (bs, hd)),
                 P.Instr(Op.ATTN_DK, 0, 0, (o["dS"], o["q"], o["dk"]), (bs, hd))]
    args = (o["q"], o["k"], o["v"], o["do"])
    prog += [P.Instr(Op.ATTN_FWD_TILED_SEG, 0, 0, (o["q"], o["k"], o["v"], o["o2"]), (o["stats"], geo, o["starts"]))
             if segments else P.Instr(Op.ATTN_FWD_TILED, 0, 0, (o["q"], o["k"], o["v"], o["o2"]), (o["stats"], bs, hd)),
             P.Instr(Op.ATTN_DQ_TILED, 0, 0, args, (o["stats"], o["dq2"], geo))]
    if d <= 256:
        prog += [
             P.Instr(Op.ATTN_DK_TILED, 0, 0, args, (o["stats"], o["dk2"], geo)),
             P.Instr(Op.ATTN_DV_TILED, 0, 0, args, (o["stats"], o["dv2"], geo))]
    return prog, arena


@pytest.mark.parametrize("segments", [0, 1], ids=["causal", "segments"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_every_instruction_from_the_oracles_bytes(shape, segments):
    _compare(*_program(*shape, segments, cached=shape[1] < 2000))


@pytest.mark.parametrize("shift", [4, 8, 12])
@pytest.mark.parametrize("shape", [(1, 64, 2, 32), (2, 130, 1, 64), (1, 65, 1, 8)], ids=lambda s: "x".join(map(str, s)))
def test_tensors_that_are_no_more_than_float_aligned(shape, shift):
    _compare(*_program(*shape, 0, cached=True, shift=shift))


def _compare(prog, arena):
    cpu, gpu = arena.copy(), arena.copy()
    ref = oracle.OracleExecutor()
    ref.bind(cpu, None)
    be = B.CudaBackend(0)
    be.bind(gpu, None)
    be.set_program(prog)
    be.begin_range(0, len(prog))
    failures = []
    for i, ins in enumerate(prog):
        ref.run(prog, None, i, i + 1)
        be.execute(i, B.StepParams(1e-3, 0.9, 0.999, 1e-8, 0.01, 0, 1))
        be.flush()
        diff = np.flatnonzero(cpu != gpu)
        if diff.size and ins.opcode in BIT_EXACT:
            failures.append(f"{P.OP_NAMES[ins.opcode]}: bits differ at byte {diff[0]}")
        elif diff.size:
            lo, hi = diff[0] // 4 * 4, diff[-1] // 4 * 4 + 4
            ok, ratio = compare(gpu[lo:hi].tobytes(), cpu[lo:hi].tobytes(), 1e-5, 1e-7)
            if not ok:
                failures.append(f"{P.OP_NAMES[ins.opcode]}: err/bound {ratio:.3g}")
        gpu[:] = cpu
        be.host_wrote(0, gpu.size)
    be.end_range()
    be.close()
    assert not failures, "\n".join(failures)
