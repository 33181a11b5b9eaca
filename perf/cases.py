"""Performance cases: the work a program that uses this package has it do, through its public calls.

What a trainer does, in the order in which it spends its time: whole LoRA training steps on one
GPU (from a test-sized model to a 3B one, equal and ragged sequence lengths, one batch or several
accumulated ones, SFT and DPO), forward-only scoring for the evaluation gate (single examples and
groups that share a prompt), and the two lower levels of the C ABI for hosts that bring their own
model loop: a frozen matmul and a linear with its adapter, on device buffers and on host buffers.

    listed()            the cases that are always timed
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call
    run(state)          one pass
    work(case)          bytes and operations that no implementation can do without
    tolerance(case)     how far a correct implementation's results may lie apart
"""
from __future__ import annotations

import ctypes as C
import random

import numpy as np
import torch

import rust_trainer_b200 as rt
from rust_trainer_b200 import objectives, packing, quants, synth
from rust_trainer_b200._lib import DT_BF16, DT_F16, DT_F32

# ------------------------------------------------------------------ the cases


def listed() -> list:
    return [
        # The smallest training step: a test-sized model, 256 tokens.  Launches and host work are all of it.
        dict(name="step-tiny-q8_0-4x64", kind="step", preset="tiny-qwen3", quant="Q8_0", n_seq=4, min_len=64, max_len=64,
             answer=0.5, rank=8, recompute=False, micro=1),
        # Qwen3-0.6B shape, Q4_0, 4 x 256: the workload that also runs on a CPU.
        dict(name="step-0.6b-q4_0-4x256", kind="step", preset="qwen3-0.6b", quant="Q4_0", n_seq=4, min_len=256, max_len=256,
             answer=0.5, rank=16, recompute=False, micro=1),
        # The headline training step: Q8_0, 16 x 512, loss on the last 30 %, activation recomputation on.
        dict(name="step-0.6b-q8_0-16x512", kind="step", preset="qwen3-0.6b", quant="Q8_0", n_seq=16, min_len=512, max_len=512,
             answer=0.3, rank=16, recompute=True, micro=1),
        # Qwen2.5-0.5B shape (64-wide heads, biases, Q4_K and Q4_0), every position a target: the head's share is largest.
        dict(name="step-0.5b-q4_k-8x1024", kind="step", preset="qwen2.5-0.5b", quant="Q4_K", n_seq=8, min_len=1024, max_len=1024,
             answer=1.0, rank=8, recompute=False, micro=1),
        # Llama-3.2-3B shape, Q6_K, sequences of 2048: the largest matmuls and the longest attention rows.
        dict(name="step-3b-q6_k-4x2048", kind="step", preset="llama-3.2-3b", quant="Q6_K", n_seq=4, min_len=2048, max_len=2048,
             answer=1.0, rank=16, recompute=False, micro=1),
        # Instruction data as it comes: examples of all lengths, four batches accumulated into one update,
        # no two of them with the same token count.
        dict(name="accumulate-0.6b-ragged", kind="step", preset="qwen3-0.6b", quant="Q8_0", n_seq=4, min_len=24, max_len=700,
             answer=0.4, rank=16, recompute=False, micro=4),
        # A DPO update on eight preference pairs: two scoring passes, then one pass over [chosen | rejected].
        dict(name="dpo-0.6b-q8_0-8-pairs", kind="dpo", preset="qwen3-0.6b", quant="Q8_0", n_seq=8, min_len=60, max_len=400,
             answer=0.5, rank=16),
        # The evaluation gate on one example: forward only, one short sequence.
        dict(name="score-0.6b-q8_0-1x157", kind="score", preset="qwen3-0.6b", quant="Q8_0", n_seq=1, min_len=157, max_len=157,
             answer=0.25, rank=16),
        # The gate on a packed group: twelve answers behind one prompt of 384 tokens.
        dict(name="score-packed-0.6b-12-of-384", kind="packed", preset="qwen3-0.6b", quant="Q8_0", n_seq=12, shared=384,
             min_len=17, max_len=90, rank=16),
        # A host that keeps its activations on the device: forward and backward of one large linear
        # with its adapter (Qwen3-4B's down projection), the adapter's gradients read back for its own optimiser.
        dict(name="linear-q4_0-2560x9728-t4096", kind="linear", quant="Q4_0", rows=2560, cols=9728, t=4096, rank=32),
        # The frozen matmul alone, few rows (a decode-sized batch): W.x and W^T.dy read the packed bytes.
        dict(name="frozen-q6_k-8192x3072-t24", kind="frozen", quant="Q6_K", rows=8192, cols=3072, t=24, act="f16", out="f32"),
        # The trait methods with host arrays in and out, at the 128 tokens the reference's own timing uses.
        dict(name="host-linear-q8_0-3072x1024-t128", kind="host_linear", quant="Q8_0", rows=3072, cols=1024, t=128, rank=8),
    ]


#: Linear shapes [out x in] of the model shapes above, for the two lower levels.
SHAPES = [(1024, 1024), (1024, 2048), (2048, 1024), (3072, 1024), (1024, 3072), (896, 896), (128, 896), (4864, 896), (896, 4864),
          (3072, 3072), (8192, 3072), (3072, 8192), (1024, 2560), (4096, 2560), (2560, 4096), (9728, 2560), (2560, 9728)]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["step", "step", "step", "step", "dpo", "score", "packed", "linear", "linear", "frozen", "frozen", "host_linear"])
    if kind in ("linear", "frozen", "host_linear"):
        rows, cols = rng.choice(SHAPES)
        quant = rng.choice([q for q in ("Q4_0", "Q8_0", "Q4_K", "Q6_K", "F16", "BF16") if cols % quants.BLOCK[quants.BY_NAME[q]][0] == 0])
        case = dict(kind=kind, quant=quant, rows=rows, cols=cols)
        if kind == "frozen":
            return dict(case, t=_log_int(rng, 1, 16384), act=rng.choice(["f16", "f16", "bf16"]), out=rng.choice(["f32", "f32", "same"]))
        return dict(case, t=_log_int(rng, 1, 512 if kind == "host_linear" else 16384), rank=rng.choice([4, 8, 16, 32, 64]))
    preset = rng.choice(["tiny-qwen3", "tiny-llama", "qwen3-0.6b", "qwen3-0.6b", "qwen3-0.6b", "qwen2.5-0.5b", "llama-3.2-3b"])
    quant = {"llama-3.2-3b": "Q6_K", "qwen2.5-0.5b": "Q4_K"}.get(preset) or rng.choice(["Q4_0", "Q8_0"])
    rank = rng.choice([8, 16])
    if kind == "packed":
        return dict(kind=kind, preset=preset, quant=quant, n_seq=rng.randint(2, 16), shared=_log_int(rng, 32, 800), min_len=8,
                    max_len=_log_int(rng, 12, 120), rank=rank)
    most = {"llama-3.2-3b": 4096, "tiny-qwen3": 2048, "tiny-llama": 2048}.get(preset, 8192)
    if kind == "score":
        n_seq = rng.choice([1, 1, 2, 5, 16])
        n = _log_int(rng, 16, min(1024, most // n_seq))
        return dict(kind=kind, preset=preset, quant=quant, n_seq=n_seq, min_len=max(4, n // 3), max_len=n, answer=0.3, rank=rank)
    tokens = _log_int(rng, 64, most // 2)
    n_seq = min(rng.choice([1, 2, 4, 8, 16]), max(1, tokens // 16))
    n = max(8, tokens // n_seq)
    ragged = rng.random() < 0.5
    case = dict(kind=kind, preset=preset, quant=quant, n_seq=n_seq, min_len=max(8, n // 4) if ragged else n, max_len=n,
                answer=rng.choice([0.3, 0.5, 1.0]), rank=rank)
    if kind == "dpo":
        return dict(case, n_seq=max(1, n_seq // 2))
    return dict(case, recompute=rng.random() < 0.4, micro=rng.choice([1, 1, 2]))


# ------------------------------------------------------------------ inputs

_CTX = None
_BLOCKS: dict = {}   # quant -> a pool of independent blocks of N(0, 0.02), made once
_TENSORS: dict = {}  # (preset, quant) -> the model file's tensors, made once: the file is the same for every run


def _ctx() -> rt.Context:
    """One context per GPU and process, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = rt.Context(0)
    return _CTX


def _packed(quant: int, rows: int, cols: int, seed: int) -> np.ndarray:
    """A [rows x cols] tensor of N(0, 0.02) as ggml stores it, from a pool of quantised blocks."""
    per = max(quants.BLOCK[quant][0], 64)  # weights a pool entry holds
    if quant not in _BLOCKS:
        w = np.random.default_rng(20240).standard_normal((1 << 15, per), dtype=np.float32) * np.float32(0.02)
        _BLOCKS[quant] = torch.from_numpy(quants.quantize(w, quant))
    pool = _BLOCKS[quant]
    if cols % per:
        raise ValueError(f"row length {cols} is not a multiple of {per}")
    pick = torch.randint(0, pool.shape[0], (rows * (cols // per),), generator=torch.Generator().manual_seed(seed))
    return pool.index_select(0, pick).reshape(rows, -1).numpy()


def _model_file(preset: str, quant: str):
    spec = synth.preset(preset, quant=quant)
    if (preset, quant) not in _TENSORS:
        T = {}

        def quantised(name, rows, cols):
            t = spec.quant_for(cols)
            T[name] = (t, rows, cols, _packed(t, rows, cols, 7 + len(T)))

        def plain(name, values):
            T[name] = (0, 1, values.size, np.ascontiguousarray(values, dtype=np.float32))

        rng = np.random.default_rng(3)
        quantised("token_embd.weight", spec.vocab, spec.hidden)
        if not spec.tie_embeddings:
            quantised("output.weight", spec.vocab, spec.hidden)
        plain("output_norm.weight", np.ones(spec.hidden))
        if spec.rope_llama3_factor > 0:
            plain("rope_freqs.weight", synth.llama3_rope_factors(spec.rot_dim, spec.rope_theta, spec.rope_llama3_factor))
        for li in range(spec.n_layers):
            p = f"blk.{li}."
            plain(p + "attn_norm.weight", 1 + 0.1 * rng.standard_normal(spec.hidden))
            plain(p + "ffn_norm.weight", 1 + 0.1 * rng.standard_normal(spec.hidden))
            if spec.qk_norm:
                plain(p + "attn_q_norm.weight", 1 + 0.1 * rng.standard_normal(spec.head_dim))
                plain(p + "attn_k_norm.weight", 1 + 0.1 * rng.standard_normal(spec.head_dim))
            for nm, (rows, cols) in spec.linear_shapes().items():
                quantised(p + nm + ".weight", rows, cols)
                if spec.attn_bias and nm in ("attn_q", "attn_k", "attn_v"):
                    plain(p + nm + ".bias", 0.01 * rng.standard_normal(rows))
        _TENSORS[preset, quant] = T
    return spec, _TENSORS[preset, quant]


def _lengths(case: dict, salt: int = 0) -> list:
    """The lengths of a batch's examples, spread over their logarithm; part of the case, not of the seed."""
    rng = random.Random(f"{case['n_seq']} {case['min_len']} {case['max_len']} {salt}")
    return [_log_int(rng, case["min_len"], case["max_len"]) for _ in range(case["n_seq"])]


def _answer_start(case: dict, n: int) -> int:
    return max(1, min(n - 1, round(n * (1 - case["answer"]))))


def _examples(case: dict, vocab: int, rng, salt: int = 0) -> list:
    return [(rng.integers(0, vocab, n, dtype=np.int32), _answer_start(case, n)) for n in _lengths(case, salt)]


class _State:
    pass


class _Memory:
    """The library's gradient buffer as torch sees it, without a copy; keeps the model that owns it."""

    def __init__(self, model):
        ptr, n = model.grad_buffer()
        self.owner = model
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3)


def _prepare_model(case: dict, seed: int):
    s = _State()
    s.case = case
    spec, tensors = _model_file(case["preset"], case["quant"])
    s.model = rt.Model(_ctx(), spec.config(), tensors)
    s.model.attach_lora(case["rank"], 2.0 * case["rank"], None, seed)
    rng = np.random.default_rng(seed)
    for lin in s.model.lora_linears():  # an adapter that has been trained for a while
        lin.write_lora(None, rng.standard_normal((lin.out_dim(), case["rank"]), dtype=np.float32) * np.float32(1e-2))
    s.grads = torch.as_tensor(_Memory(s.model), device="cuda:0")
    if case["kind"] == "step":
        if case["recompute"]:
            s.model.set_checkpointing(1)
        s.batches = [_examples(case, spec.vocab, rng, k) for k in range(case["micro"])]
    elif case["kind"] == "dpo":
        s.pairs = list(zip(_examples(case, spec.vocab, rng, 1), _examples(case, spec.vocab, rng, 2)))
        s.ref = objectives.dpo_ref_logps(s.model, s.pairs)
    elif case["kind"] == "score":
        s.seqs, s.tpos, s.ttok, _ = objectives._layout(_examples(case, spec.vocab, rng))
    else:
        prompt = rng.integers(0, spec.vocab, case["shared"], dtype=np.int32)
        seqs = [np.concatenate([prompt, [i], rng.integers(0, spec.vocab, n, dtype=np.int32)]).astype(np.int32) for i, n in enumerate(_lengths(case))]
        s.group = packing.pack(seqs)
        at = [s.group.map_targets(k, *synth.answer_targets(q, case["shared"] + 1)) for k, q in enumerate(seqs)]
        s.tpos, s.ttok = np.concatenate([a for a, _ in at]), np.concatenate([b for _, b in at])
    return s


def _prepare_linear(case: dict, seed: int):
    s = _State()
    s.case = case
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    t, rows, cols = case["t"], case["rows"], case["cols"]
    q = quants.BY_NAME[case["quant"]]
    s.frozen = rt.Frozen(_ctx(), q, rows, cols, _packed(q, rows, cols, seed))
    x = torch.randn(t, cols, generator=g, device="cuda:0")
    # gradients whose rows differ in size by a few powers of ten, as they do between tokens
    dy = torch.randn(t, rows, generator=g, device="cuda:0") * torch.exp(torch.randn(t, 1, generator=g, device="cuda:0")) * 1e-3
    if case["kind"] != "frozen":
        rng = np.random.default_rng(seed)
        r = case["rank"]
        s.lin = rt.Linear("linear", s.frozen)
        s.lin.attach_lora(r, 2.0 * r, rng.standard_normal((r, cols), dtype=np.float32) / np.float32(r),
                          rng.standard_normal((rows, r), dtype=np.float32) * np.float32(1e-2))
        s.ga, s.gb = torch.empty(r, cols).pin_memory(), torch.empty(rows, r).pin_memory()
    if case["kind"] == "host_linear":
        s.x, s.dy = x.cpu().numpy(), dy.cpu().numpy()
        return s
    act = torch.bfloat16 if case.get("act") == "bf16" else torch.float16
    out = act if case.get("out") == "same" else torch.float32
    s.x = x.to(act)
    if case["kind"] == "linear":
        s.scale = dy.abs().amax(1).contiguous()
        s.dy = (dy / s.scale[:, None]).to(act)
        s.y = torch.empty(t, rows, dtype=torch.float16, device="cuda:0")
        s.dx = torch.empty(t, cols, dtype=torch.float32, device="cuda:0")
    else:
        s.dy = (dy * 1e3).to(act)
        s.y, s.dx = torch.empty(t, rows, dtype=out, device="cuda:0"), torch.empty(t, cols, dtype=out, device="cuda:0")
    torch.cuda.synchronize()
    return s


def prepare(case: dict, seed: int):
    return (_prepare_linear if case["kind"] in ("linear", "frozen", "host_linear") else _prepare_model)(case, seed)


# ------------------------------------------------------------------ one pass

_DT = {torch.float32: DT_F32, torch.bfloat16: DT_BF16, torch.float16: DT_F16}


def _p(t: torch.Tensor):
    return C.c_void_p(t.data_ptr())


def _f(t: torch.Tensor):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def _run_step(s):
    s.model.zero_grad()
    losses = [objectives.sft_batch_grad(s.model, b) for b in s.batches]
    norm = s.model.optim_step(5e-5, 1.0, weight_decay=0.01)  # the next pass runs on the updated adapters
    return dict(losses=losses, norm=norm, grads=s.grads)


def _run_dpo(s):
    s.model.zero_grad()
    loss = objectives.dpo_batch_grad(s.model, s.pairs, s.ref, 0.1)
    norm = s.model.optim_step(5e-5, 1.0, weight_decay=0.01)
    return dict(loss=loss, norm=norm, grads=s.grads)


def _run_score(s):
    logp, hits, _ = s.model.score(s.seqs, s.tpos, s.ttok)
    return dict(logp=logp, hits=hits)


def _run_packed(s):
    logp, hits = s.model.score_packed([s.group], s.tpos, s.ttok)
    return dict(logp=logp, hits=hits)


def _run_linear(s):
    L, lin, ctx, t = rt.lib(), s.lin._h, s.frozen.ctx, s.case["t"]
    s.lin.zero_grad()
    ctx.check(L.rt_linear_forward_dev(lin, _p(s.x), t, _p(s.y), DT_F16, 0))
    ctx.check(L.rt_linear_backward_dev(lin, _p(s.x), _p(s.dy), _p(s.scale), t, _p(s.dx), 0))
    ctx.check(L.rt_lora_read(lin, None, None, _f(s.ga), _f(s.gb)))
    return dict(y=s.y, dx=s.dx, ga=s.ga, gb=s.gb)


def _run_frozen(s):
    L, w, ctx, t = rt.lib(), s.frozen._h, s.frozen.ctx, s.case["t"]
    ctx.check(L.rt_frozen_forward_dev(w, _p(s.x), _DT[s.x.dtype], t, _p(s.y), _DT[s.y.dtype], 0))
    ctx.check(L.rt_frozen_backward_input_dev(w, _p(s.dy), _DT[s.dy.dtype], t, _p(s.dx), _DT[s.dx.dtype], 0))
    return dict(y=s.y, dx=s.dx)


def _run_host_linear(s):
    t = s.case["t"]
    s.lin.zero_grad()
    y = s.lin.forward(s.x, t)
    dx = s.lin.backward(s.x, s.dy, t)
    s.frozen.ctx.check(rt.lib().rt_lora_read(s.lin._h, None, None, _f(s.ga), _f(s.gb)))
    return dict(y=y, dx=dx, ga=s.ga, gb=s.gb)


_RUN = dict(step=_run_step, dpo=_run_dpo, score=_run_score, packed=_run_packed, linear=_run_linear, frozen=_run_frozen, host_linear=_run_host_linear)


def run(s):
    return _RUN[s.case["kind"]](s)


# ------------------------------------------------------------------ what a pass cannot do without


def _model_work(case: dict):
    spec = synth.preset(case["preset"], quant=case["quant"])
    weights = [(r, c) for r, c in spec.linear_shapes().values()]
    params = spec.n_layers * sum(r * c for r, c in weights)
    nbytes = spec.n_layers * sum(r * quants.row_bytes(spec.quant_for(c), c) for r, c in weights)
    head_bytes = spec.vocab * quants.row_bytes(spec.quant_for(spec.hidden), spec.hidden)
    lora = spec.n_layers * case["rank"] * sum(r + c for r, c in weights)
    qd = spec.n_heads * spec.head_dim * spec.n_layers

    def passes(lengths, shared, targets, backward):
        """Operations and host bytes of one pass; a token of an example also sees the shared prompt."""
        tokens = shared + sum(lengths)
        pairs = shared * (shared + 1) / 2 + sum(n * (n + 1) / 2 + n * shared for n in lengths)
        fwd = 2 * tokens * (params + lora) + 4 * qd * pairs + 2 * targets * spec.vocab * spec.hidden
        bwd = 2 * tokens * (params + 2 * lora) + 10 * qd * pairs + 2 * targets * spec.vocab * spec.hidden
        return fwd + (bwd if backward else 0), 12 * tokens + 12 * targets

    kind = case["kind"]
    flops = io = 0
    if kind == "packed":
        own = [n + 1 for n in _lengths(case)]
        flops, io = passes(own, case["shared"], sum(own) - len(own), False)
    elif kind == "score":
        ls = _lengths(case)
        flops, io = passes(ls, 0, sum(n - _answer_start(case, n) for n in ls), False)
    else:
        for salt in range(case["micro"]) if kind == "step" else (1, 2):
            ls = _lengths(case, salt)
            f, b = passes(ls, 0, sum(n - _answer_start(case, n) for n in ls), True)
            flops, io = flops + f, io + b
    update = 4 * 7 * lora if kind in ("step", "dpo") else 4 * lora  # A and B, their gradients, Adam's m and v: read and written
    return dict(bytes=nbytes + head_bytes + update + io, flops=flops)


def work(case: dict) -> dict:
    if "preset" in case:
        return _model_work(case)
    t, rows, cols, r = case["t"], case["rows"], case["cols"], case.get("rank", 0)
    weight = rows * quants.row_bytes(quants.BY_NAME[case["quant"]], cols)
    flops = 4 * t * rows * cols + 6 * t * r * (rows + cols)
    if case["kind"] == "host_linear":
        return dict(bytes=weight + 8 * t * (rows + cols) + 8 * r * (rows + cols), flops=flops)
    e = 2 if case["kind"] == "linear" or case["out"] == "same" else 4
    y, dx = (2, 4) if case["kind"] == "linear" else (e, e)
    return dict(bytes=weight + 2 * t * (rows + cols) + y * t * rows + dx * t * cols + 12 * r * (rows + cols) + (4 * t if r else 0), flops=flops)


def tolerance(case: dict):
    if case["kind"] == "frozen" and case["act"] == "bf16":
        return dict(rel=1e-2, max=0.1)  # weights and results rounded to 8 bits of mantissa
    if case["kind"] in ("linear", "frozen", "host_linear"):
        # 16-bit operands (11 bits), f32 sums; the largest of millions of values lies further off than their norm
        return dict(rel=2e-3, max=0.05)
    if case["kind"] in ("score", "packed"):
        return dict(rel=1e-3, max=1e-2)  # log-probabilities of a stack of layers on 11-bit activations
    return dict(rel=1e-2, max=0.5)  # gradients through the same stack, forward and backward
