"""Performance cases of the update-plan executor.

A case is one call (or one short sequence of calls) a user's program makes through the public entry
points, at one size.  Six kinds of work, which together are what the framework is used for:

  step       one optimizer step of a LoRA update plan through the engine: `Engine.train_step` with the
             batch in host memory (staging, forward, backward, AdamW, the loss read back), ranges replayed
             as CUDA graphs.  Models: feed-forward, f32 decoder, int8-weight decoder.
  seam       the same step through the executor seam in its default (strict) coherence, as a host engine
             drives it: the batch written into the host arena and announced, the train program run, every
             written range back in the host arena.
  evaluate   `Engine.evaluate_rows`: the forward program in f32 arithmetic, the loss, the accuracy tally and
             the real-row loss of a batch whose last rows are padding.
  merge      `Engine.run_merge`: every adapter's weight delta and its finiteness scan, before a commit.
  gemm       the training step around one square frozen weight with an adapter, as an instruction program
             through the seam in lazy coherence; f32 and relaxed (bf16 tensor core) forms.
  attention  the tiled causal attention chain (forward, dQ, dK, dV), relaxed, through the seam.

Training cases start from a checkpoint in the middle of a run (non-zero adapters and moments), as a
resumed job does; the inputs of a pass come from the seed, the frozen weights from the configuration.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from see_ai_b200 import backend as B
from see_ai_b200 import plan as P
from see_ai_b200 import synth
from see_ai_b200 import workloads as W
from see_ai_b200.engine import Engine

RESUMED_AT = 200   # the optimizer timestep of the checkpoint the training cases resume from


# ---- the cases --------------------------------------------------------------------------------------

def _mlp(kind, dims, batch, rank):
    return dict(kind=kind, model="mlp", dims="x".join(str(d) for d in dims), batch=batch, rank=rank)


def _decoder(kind, layers, d_model, heads, vocab, seq, seqs, rank, targets, int8, attention, real_rows=0):
    return dict(kind=kind, model="decoder", layers=layers, d_model=d_model, heads=heads, ffn=4 * d_model, vocab=vocab,
                seq=seq, seqs=seqs, rank=rank, targets=targets, int8=int8, attention=attention, real_rows=real_rows)


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # The smallest step: the benchmark's feed-forward plan, 32 samples.  Launches and round trips.
        named("mlp_b32", _mlp("step", (256, 1024, 64), 32, 8)),
        # A host engine behind the seam with the default coherence; odd batch, ten classes.
        named("mlp_seam_b57", _mlp("seam", (784, 128, 10), 57, 8)),
        # The benchmark's f32 decoder at its stated size: many small f32 kernels.
        named("decoder_f32", _decoder("step", 4, 256, 4, 4096, 128, 32, 8, "qv", False, "cached")),
        # The headline: the 12-layer int8 decoder, 64 sequences of 512 on one GPU.
        named("decoder_int8_64seq", _decoder("step", 12, 768, 12, 32000, 512, 64, 16, "qkvo", True, "tiled")),
        # One rank's share of the same batch over eight GPUs.
        named("decoder_int8_8seq", _decoder("step", 12, 768, 12, 32000, 512, 8, 16, "qkvo", True, "tiled")),
        # A short ragged fine-tune: three sequences of 200 tokens, adapters on Q and V only.
        named("decoder_int8_ragged", _decoder("step", 4, 512, 8, 8000, 200, 3, 8, "qv", True, "tiled")),
        # Validation of the f32 decoder, the last batch partly padding.
        named("eval_f32", _decoder("evaluate", 4, 256, 4, 4096, 128, 32, 8, "qv", False, "cached", 4000)),
        # Validation of the int8 decoder before and after an update (what the commit gate reads).
        named("eval_int8_8seq", _decoder("evaluate", 12, 768, 12, 32000, 512, 8, 16, "qkvo", True, "tiled", 4096)),
        # The deltas of all 48 adapters of that decoder, for the commit.
        named("merge_int8", _decoder("merge", 12, 768, 12, 32000, 512, 8, 16, "qkvo", True, "tiled")),
        # The middle of the GEMM sweep, in both arithmetics.
        named("gemm_f32_2048", dict(kind="gemm", S=2048, rank=8, relaxed=False)),
        named("gemm_bf16_4096", dict(kind="gemm", S=4096, rank=8, relaxed=True)),
        # The middle of the attention sweep.
        named("attention_s2048_d64", dict(kind="attention", Bq=8, S=2048, H=16, d=64)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step_mlp", "seam", "step_f32", "step_int8", "step_int8", "evaluate", "merge", "gemm", "attention"))
    rank = rng.choice((4, 8, 16))
    targets = rng.choice(("qv", "qkvo", "q", "qkv"))
    if kind in ("step_mlp", "seam"):
        dims = [_log(rng, 32, 1024) for _ in range(rng.choice((2, 3)))] + [_log(rng, 4, 512)]
        return _mlp("seam" if kind == "seam" else "step", dims, _log(rng, 1, 512), rank)
    f32 = kind == "step_f32" or (kind == "evaluate" and rng.random() < 0.5)
    if f32:
        d_model = rng.choice((128, 192, 256, 384))
        seq = _log(rng, 16, 256)
        return _decoder("evaluate" if kind == "evaluate" else "step", rng.randint(1, 4), d_model, d_model // rng.choice((32, 64)),
                        _log(rng, 256, 8192), seq, max(1, min(64, _log(rng, 64, 4096) // seq)), rank, targets, False,
                        rng.choice(("cached", "tiled")), _log(rng, 1, 4096) if kind == "evaluate" else 0)
    if kind in ("step_int8", "evaluate", "merge"):
        d_model = rng.choice((256, 512, 768))
        vocab, seq, rows = _log(rng, 1000, 16000), _log(rng, 64, 512), _log(rng, 128, 8192 if kind == "step_int8" else 2048)
        if rng.random() < 0.75:   # tokenizers mostly pad their vocabularies, batches are mostly cut to a round length
            vocab, seq = (vocab + 63) // 64 * 64, (seq + 7) // 8 * 8
        return _decoder(kind.replace("_int8", ""), rng.randint(1, 4), d_model, d_model // 64, vocab, seq, max(1, rows // seq), rank,
                        targets, True, "tiled", _log(rng, 1, 2048) if kind == "evaluate" else 0)
    if kind == "gemm":
        S = _log(rng, 256, 4096)
        return dict(kind="gemm", S=S if S < 1024 and rng.random() < 0.3 else (S + 7) // 8 * 8, rank=rng.choice((8, 16)),
                    relaxed=rng.random() < 0.5)
    S = _log(rng, 64, 4096) // 8 * 8
    return dict(kind="attention", Bq=max(1, min(16, 16384 // S)), S=S, H=rng.choice((8, 12, 16)), d=rng.choice((64, 128)))


# ---- plans and programs (kept: a user's program builds its plan once) --------------------------------

@functools.lru_cache(maxsize=4)
def _plan(model, dims, batch, rank, layers, d_model, heads, ffn, vocab, seq, seqs, targets, int8, attention):
    if model == "mlp":
        blob = synth.build_mlp_plan(synth.MlpConfig(dims=tuple(int(d) for d in dims.split("x")), batch=batch, rank=rank,
                                                    alpha=2.0 * rank))
    else:
        blob = synth.build_decoder_plan(synth.DecoderConfig(
            layers=layers, d_model=d_model, heads=heads, ffn=ffn, vocab=vocab, seq=seq, batch_seqs=seqs, rank=rank,
            alpha=2.0 * rank, targets=tuple(targets), quantized=int8, attention=attention))
    return blob, P.Plan(blob)


def _plan_of(case):
    keys = ("model", "dims", "batch", "rank", "layers", "d_model", "heads", "ffn", "vocab", "seq", "seqs", "targets", "int8",
            "attention")
    return _plan(*(case.get(k) for k in keys))


@functools.lru_cache(maxsize=2)
def _program(kind, S, rank, relaxed, Bq, H, d):
    prog = W.gemm_step_program(S, relaxed, rank) if kind == "gemm" else W.attention_chain_program(Bq, S, H, d, relaxed=True)
    return prog, P.pack_program(prog.instrs)


# ---- device views: tensors over an arena, which stays alive as long as they do ------------------------

class _Bytes:
    def __init__(self, owner, pointer, nbytes):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(nbytes // 4,), typestr="<f4", data=(pointer, False), version=3)


def _view(owner, backend, offset, nbytes):
    return torch.as_tensor(_Bytes(owner, backend.device_arena() + offset, nbytes), device="cuda")


# ---- inputs -------------------------------------------------------------------------------------------

def _checkpoint(plan, rng):
    """The persistent prefix in the middle of a run: adapters that have moved, AdamW moments of the size
    the gradients have."""
    state = np.frombuffer(plan.persist_init, dtype=np.uint8).copy().view(np.float32)
    for ins in plan.train:
        if ins.opcode != P.Op.ADAMW_STEP:
            continue
        n = ins.out[0]
        p, m, v = (state[ins.ins[i] // 4:ins.ins[i] // 4 + n] for i in (0, 2, 3))
        p += rng.standard_normal(n, dtype=np.float32) * np.float32(0.02)
        m[:] = rng.standard_normal(n, dtype=np.float32) * np.float32(3e-5)
        v[:] = np.square(rng.standard_normal(n, dtype=np.float32)) * np.float32(1e-8) + np.float32(1e-9)
    return state


def _batch(case, plan, rng):
    rows = plan.header["batch"]
    if case["model"] == "mlp":
        dims = [int(d) for d in case["dims"].split("x")]
        return (rng.standard_normal((rows, dims[0]), dtype=np.float32), rng.integers(0, dims[-1], size=rows, dtype=np.int32))
    record = rng.integers(0, case["vocab"], size=(case["seqs"], case["seq"] + 1), dtype=np.int32)
    return (np.ascontiguousarray(record[:, :-1]).reshape(-1), np.ascontiguousarray(record[:, 1:]).reshape(-1))


def _gradient_block(plan):
    spans = [(i.ins[1], i.ins[1] + 4 * i.out[0]) for i in plan.train if i.opcode == P.Op.ADAMW_STEP]
    lo, hi = min(s[0] for s in spans), max(s[1] for s in spans)
    return lo, hi - lo


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("gemm", "attention"):
        prog, code = _program(kind, case["S"], case.get("rank"), case.get("relaxed"), case.get("Bq"), case.get("H"), case.get("d"))
        be = B.CudaBackend(0)
        be.set_coherence(B.COHERENCE_LAZY)
        be.bind(prog.arena, prog.rodata)
        be.set_program(code)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        if kind == "gemm":
            S, r = case["S"], case["rank"]
            sizes = dict(A=(S * S, 1.0), dC=(S * S, 1.0), La=(S * r, S ** -0.5), Lb=(S * r, 0.02))
            outs = dict(C=S * S, dA=S * S, dW=S * S, dLa=S * r, dLb=S * r)
        else:
            n = case["Bq"] * case["S"] * case["H"] * case["d"]
            sizes = {k: (n, 1.0) for k in ("q", "k", "v", "do")}
            outs = {k: n for k in ("o", "dq", "dk", "dv")}
        for name, (n, scale) in sizes.items():
            _view(be, be, prog.refs[name], 4 * n).copy_(torch.randn(n, generator=gen, device="cuda") * scale)
        torch.cuda.synchronize()
        return dict(kind=kind, backend=be, outputs={k: _view(be, be, prog.refs[k], 4 * n) for k, n in outs.items()})

    blob, plan = _plan_of(case)
    rng = np.random.default_rng(seed)
    x, y = _batch(case, plan, rng)
    checkpoint = _checkpoint(plan, rng)
    h = plan.header
    g_off, g_bytes = _gradient_block(plan)
    if kind == "seam":
        arena = plan.stage_arena()
        arena[:checkpoint.nbytes] = checkpoint.view(np.uint8)
        be = B.CudaBackend(0)
        be.bind(arena, np.frombuffer(plan.rodata, dtype=np.uint8).copy())
        be.set_program(P.pack_program(plan.train))
        params = B.StepParams(h["lr"], h["beta1"], h["beta2"], h["eps"], h["weight_decay"], 0, RESUMED_AT + 1)
        slots = [(h["input_ref"], x.view(np.uint8).reshape(-1)), (h["label_ref"], y.view(np.uint8).reshape(-1))]
        outputs = dict(loss=arena[h["loss_ref"]:h["loss_ref"] + 4].view(np.float32),
                       gradients=arena[g_off:g_off + g_bytes].view(np.float32),
                       persistent=arena[:h["persistent_size"]].view(np.float32))
        return dict(kind=kind, backend=be, arena=arena, slots=slots, params=params, outputs=outputs)

    eng = Engine(0)
    eng.load(blob)
    eng.set_use_graphs(True)
    eng.set_horizon(h["default_steps"])
    eng.restore(checkpoint.view(np.uint8), RESUMED_AT)
    state = dict(kind=kind, engine=eng, x=x, y=y)
    if kind == "step":
        state["outputs"] = dict(gradients=_view(eng, eng.backend, g_off, g_bytes),
                                persistent=_view(eng, eng.backend, 0, h["persistent_size"]))
    elif kind == "evaluate":
        state["real_rows"] = min(case["real_rows"], h["batch"])
        loss = next(i for i in plan.eval if i.opcode == P.Op.XENT_FWD)
        state["outputs"] = dict(probabilities=_view(eng, eng.backend, loss.ins[3], 4 * loss.out[0] * loss.out[1]))
    else:
        lo = min(e.arena_offset for e in plan.emit)
        hi = max(e.arena_offset + e.byte_size for e in plan.emit)
        state["outputs"] = dict(deltas=_view(eng, eng.backend, lo, hi - lo))
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        loss = state["engine"].train_step(state["x"], state["y"])
        return dict(state["outputs"], loss=loss)
    if kind == "seam":
        arena, be = state["arena"], state["backend"]
        for offset, data in state["slots"]:
            arena[offset:offset + data.size] = data
            be.host_wrote(offset, data.size)
        be.run(params=state["params"])
        return state["outputs"]
    if kind == "evaluate":
        r = state["engine"].evaluate_rows(state["x"], state["y"], state["real_rows"])
        return dict(state["outputs"], loss=float(r.loss), rows=int(r.rows), correct=int(r.correct),
                    real_row_loss=float(r.real_row_loss), loss_rows=int(r.loss_rows))
    if kind == "merge":
        finite = state["engine"].run_merge()
        return dict(state["outputs"], finite=finite)
    state["backend"].run()
    return state["outputs"]


# ---- what a pass cannot do without ---------------------------------------------------------------------

def _mlp_work(case):
    dims = [int(d) for d in case["dims"].split("x")]
    M, r = case["batch"], case["rank"]
    flops = bytes_ = 0.0
    for i, (k, n) in enumerate(zip(dims, dims[1:])):
        flops += 2.0 * M * k * n * (2 if i else 1) + 2.0 * M * r * (k + n) * 3 - (0 if i else 2.0 * M * r * k)
        bytes_ += 4.0 * k * n + 4.0 * n + 28.0 * r * (k + n)     # frozen weight, bias; AdamW reads 4 and writes 3 arrays
    return flops, bytes_ + 4.0 * M * (dims[0] + 1)


def _decoder_work(case, train):
    L, D, F, V, S, n, r = (case[k] for k in ("layers", "d_model", "ffn", "vocab", "seq", "seqs", "rank"))
    M, sites = float(n * S), len(case["targets"])
    weights = L * (4 * D * D + 2 * D * F) + D * V
    pairs = n * case["heads"] * (S * (S + 1) / 2.0)              # causal (query, key) pairs
    flops = 2.0 * M * weights + L * (4.0 * pairs * (D // case["heads"]) + 4.0 * M * D * r * sites)
    bytes_ = weights * (1.0 if case["int8"] else 4.0) + M * 4.0 * D + 8.0 * M
    if train:   # input gradients (layer 0's projections need none), attention backward, the adapters' products
        flops += 2.0 * M * (weights - 3 * D * D) + L * (10.0 * pairs * (D // case["heads"]) + 8.0 * M * D * r * sites)
        bytes_ += 28.0 * L * sites * 2 * D * r
    else:
        bytes_ += 4.0 * L * sites * 2 * D * r
    return flops, bytes_


def work(case):
    kind = case["kind"]
    if kind in ("step", "seam", "evaluate"):
        flops, bytes_ = _mlp_work(case) if case["model"] == "mlp" else _decoder_work(case, kind != "evaluate")
    elif kind == "merge":
        L, D, r, sites = case["layers"], case["d_model"], case["rank"], len(case["targets"])
        flops, bytes_ = 2.0 * L * sites * D * D * r, L * sites * (4.0 * D * D + 8.0 * D * r)
    elif kind == "gemm":
        S, r = case["S"], case["rank"]
        flops = 3 * 2.0 * S ** 3 + 6 * 2.0 * S * S * r
        bytes_ = 4.0 * (3 * S * S + 3 * S * S + 6 * S * r)
    else:
        pairs = case["Bq"] * case["H"] * (case["S"] * (case["S"] + 1) / 2.0)
        flops = (4.0 + 10.0) * pairs * case["d"]
        bytes_ = 4.0 * 8 * case["Bq"] * case["S"] * case["H"] * case["d"]
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Relaxed instructions round activations, probabilities and gradients to bf16 on the way (2^-9 each, a
    # few dozen times along a decoder's backward); everything else is f32 arithmetic in another order.
    if case["kind"] == "attention" or (case["kind"] == "gemm" and case["relaxed"]) or (case["kind"] == "step" and case.get("int8")):
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 1e-5, "max": 1e-3}
