"""Performance cases: what a training or serving program has the framework do on one GPU, through its public entry points.

Paths (field ``path``):

* ``sft``      one optimizer step of full fine-tuning, ``TrainEngine.sft_step`` once per micro-batch of the window;
* ``lora``     the same with LoRA adapters on all projections of a frozen base;
* ``grpo``     one GRPO step, ``TrainEngine.grpo_step``, over groups of sampled responses of unequal length, with a frozen
  reference policy and the KL term;
* ``prefill``  prompts into the paged cache, ``InferenceEngine.feed`` in chunks, logits of each prompt's last token;
* ``decode``   one token for every running sequence: ``prepare_decode`` and a replay of the captured decode step, as the
  engine does with ``enable_cuda_graph``.

Weights are random, at the scale of the presets' initialisation but for the dense models' output projections: those are small
enough for every sublayer to add little to the residual stream, as in a trained model (at the initialisation's scale the sublayers
of a random model outweigh the stream and amplify each rounding many times over).  Tokens are uniform over the vocabulary.
"""
import gc
import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

DENSE = {
    # hidden, layers, heads, kv heads, feed-forward (head size 128, vocabulary 151936, tied embedding)
    "qwen3-0.6b": (1024, 28, 16, 8, 3072),
    "qwen3-4b": (2560, 36, 32, 8, 9728),
}
VOCAB, HEAD, EPS, THETA = 151936, 128, 1e-6, 1e6
SOTAZEN = {"sotazen-0.6b": dict(width=1024, heads=8, depth=28, ff=5120, kv_heads=4, window=1024, rank=512, rot=64)}
LORA_RANK, LORA_ALPHA = 16, 32.0
LR, WD, BETA1, BETA2, ADAM_EPS, CLIP = 1e-5, 0.01, 0.9, 0.999, 1e-8, 1.0
KL_BETA, CLIP_EPS = 0.1, 0.2


# ---- the cases -------------------------------------------------------------------------------------------------------
def listed():
    return [
        # fine-tuning on single short examples: launches and the optimizer count
        {"name": "sft_1x256", "path": "sft", "model": "qwen3-0.6b", "batch": 1, "seq": 256, "accum": 1},
        # the headline training step: micro-batch 8 x 1024, two micro-batches per optimizer step
        {"name": "sft_8x1024", "path": "sft", "model": "qwen3-0.6b", "batch": 8, "seq": 1024, "accum": 2},
        # long examples of an odd length: attention weighs more, the last tile is ragged
        {"name": "sft_4x2047", "path": "sft", "model": "qwen3-0.6b", "batch": 4, "seq": 2047, "accum": 1},
        # adapters on the larger model
        {"name": "lora_4b_4x1024", "path": "lora", "model": "qwen3-4b", "batch": 4, "seq": 1024, "accum": 1},
        # a chunk of a reinforcement-learning batch: 2 prompts x 8 samples, 256 + up to 512 tokens
        {"name": "grpo_2x8x768", "path": "grpo", "model": "qwen3-0.6b", "prompts": 2, "samples": 8, "prompt": 256, "response": 512},
        # an interactive user's long prompt, in the engine's chunks
        {"name": "prefill_1x8192", "path": "prefill", "model": "qwen3-0.6b", "batch": 1, "seq": 8192, "chunk": 2048},
        # many short prompts of unequal lengths arriving together, on the larger model
        {"name": "prefill_4b_16x300", "path": "prefill", "model": "qwen3-4b", "batch": 16, "seq": 300, "chunk": 2048},
        # one user: the latency of a token
        {"name": "decode_1x1024", "path": "decode", "model": "qwen3-0.6b", "batch": 1, "context": 1024, "kv": "fp16"},
        # the rollout / serving batch
        {"name": "decode_256x1024", "path": "decode", "model": "qwen3-0.6b", "batch": 256, "context": 1024, "kv": "fp16"},
        # a medium batch of longer contexts on the larger model, with the fp8 cache
        {"name": "decode_4b_32x2000_fp8", "path": "decode", "model": "qwen3-4b", "batch": 32, "context": 2000, "kv": "fp8"},
        # the hybrid designs: prompts and decoding of the one whose layers share kernels with the others
        {"name": "sotazen_prefill_4x2048", "path": "prefill", "model": "sotazen-0.6b", "batch": 4, "seq": 2048, "chunk": 2048},
        {"name": "sotazen_decode_64x1024", "path": "decode", "model": "sotazen-0.6b", "batch": 64, "context": 1024, "kv": "fp16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["sft", "sft", "lora", "grpo", "prefill", "prefill", "decode", "decode", "decode"])
    if path in ("sft", "lora"):
        model = "qwen3-4b" if path == "lora" and rng.random() < 0.5 else "qwen3-0.6b"
        accum = rng.choice([1, 2]) if path == "sft" else 1
        seq = _log(rng, 100, 2048)
        most = max(1, (3500 if model == "qwen3-4b" else 14000) // (seq * accum))
        return {"path": path, "model": model, "batch": rng.randint(1, min(16, most)), "seq": seq, "accum": accum}
    if path == "grpo":
        prompt, response = _log(rng, 32, 256), _log(rng, 64, 512)
        samples = rng.choice([4, 8])
        most = max(1, 12288 // (samples * (prompt + response)))
        return {"path": path, "model": "qwen3-0.6b", "prompts": rng.randint(1, min(4, most)), "samples": samples, "prompt": prompt,
                "response": response}
    model = rng.choice(["qwen3-0.6b", "qwen3-0.6b", "qwen3-4b", "sotazen-0.6b"])
    if path == "prefill":
        seq = _log(rng, 48, 8192)
        most = max(1, (5000 if model == "qwen3-4b" else 16384) // seq)
        return {"path": path, "model": model, "batch": _log(rng, 1, min(32, most)), "seq": seq, "chunk": rng.choice([1024, 2048])}
    context = _log(rng, 64, 8192)
    most = max(1, {"qwen3-0.6b": 262144, "qwen3-4b": 100000, "sotazen-0.6b": 65536}[model] // context)
    batch = _log(rng, 1, min(256, most))
    kv = "fp8" if model != "sotazen-0.6b" and rng.random() < 0.33 else "fp16"
    return {"path": path, "model": model, "batch": batch, "context": context, "kv": kv}


# ---- inputs, from the seed alone --------------------------------------------------------------------------------------
def _gen(seed, *what):
    key = 1469598103934665603
    for c in f"{seed}:{what}".encode():
        key = ((key ^ c) * 1099511628211) % (1 << 62)
    return torch.Generator(device="cuda").manual_seed(key)


def _normal(shape, std, seed, *what):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, std, generator=_gen(seed, *what))


def _ints(lo, hi, shape, seed, *what):
    return torch.randint(lo, hi, shape, generator=_gen(seed, *what), device="cuda")


def _dense_shapes(model):
    """Parameter name -> shape, in the order of the model's parameters."""
    h, layers, heads, kv, ff = DENSE[model]
    out = {"embed_tokens": (VOCAB, h)}
    for i in range(layers):
        p = f"layers.{i}."
        out |= {p + "input_layernorm.weight": (h,), p + "self_attn.qkv_proj.weight": ((heads + 2 * kv) * HEAD, h),
                p + "self_attn.o_proj.weight": (h, heads * HEAD), p + "self_attn.q_norm.weight": (HEAD,),
                p + "self_attn.k_norm.weight": (HEAD,), p + "post_attention_layernorm.weight": (h,),
                p + "mlp.gate_up_proj.weight": (2 * ff, h), p + "mlp.down_proj.weight": (h, ff)}
    out["norm.weight"] = (h,)
    return out


def _dense_weight(name, shape, seed):
    std = 0.1 if len(shape) == 1 else 0.02
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        small = shape[0] <= 1024
        std = (0.003 if small else 0.0015) if name.endswith("o_proj.weight") else (0.0002 if small else 0.00005)
    t = _normal(shape, std, seed, name)
    return ((t + 1.0) if len(shape) == 1 else t).to(torch.bfloat16)


def _adapter_shapes(model):
    """LoRA adapters: (layer, projection) -> (fused projection, rows of it, in, out), in the order of the model's parameters."""
    h, layers, heads, kv, ff = DENSE[model]
    out = {}
    for i in range(layers):
        at = 0
        for n, rows in (("q_proj", heads * HEAD), ("k_proj", kv * HEAD), ("v_proj", kv * HEAD)):
            out[(i, n)] = ("qkv_proj", slice(at, at + rows), h, rows)
            at += rows
        out[(i, "o_proj")] = ("o_proj", slice(0, h), heads * HEAD, h)
        out[(i, "gate_proj")] = ("gate_up_proj", slice(0, ff), h, ff)
        out[(i, "up_proj")] = ("gate_up_proj", slice(ff, 2 * ff), h, ff)
        out[(i, "down_proj")] = ("down_proj", slice(0, h), ff, h)
    return out


def _adapter(i, n, leaf, shape, seed):
    return _normal(shape, 0.02 if leaf == "A" else 0.002, seed, i, n, leaf)


def _sotazen_layers(model):
    c = SOTAZEN[model]
    for i in range(c["depth"]):
        yield i, "latent" if i % 4 == 3 else ("differential" if i % 4 == 2 else "lightning")


def _sotazen_weight(name, shape, seed):
    last = name.rsplit(".", 1)[-1]
    if last.startswith("norm"):
        return (1.0 + _normal(shape, 0.1, seed, name)).to(torch.bfloat16)
    std = 0.1 if last in ("lq1", "lk1", "lq2", "lk2", "b", "sink") else 0.02
    return _normal(shape, std, seed, name).to(torch.bfloat16)


def _lengths(n, hi, seed):
    """Unequal lengths around the upper half of the range; a single sequence has the full one."""
    return [hi] if n == 1 else [int(x) for x in _ints(max(1, hi // 2), hi + 1, (n,), seed, "lengths").tolist()]


def _prompts(case, seed):
    return [_ints(0, VOCAB, (n,), seed, "prompt", i).tolist()
            for i, n in enumerate(_lengths(case["batch"], case["seq" if case["path"] == "prefill" else "context"], seed))]


def _sft_batches(case, seed):
    """Per micro-batch (prompts, responses): the second half of every example is supervised."""
    half, out = case["seq"] // 2, []
    for k in range(case["accum"]):
        ids = _ints(0, VOCAB, (case["batch"], case["seq"]), seed, "batch", k).tolist()
        out.append(([r[:half] for r in ids], [r[half:] for r in ids]))
    return out


def _grpo_batch(case, seed):
    n, k, r = case["prompts"], case["samples"], case["response"]
    prompts = _ints(0, VOCAB, (n, case["prompt"]), seed, "prompts").tolist()
    lens = _ints(max(1, r // 4), r + 1, (n, k), seed, "lengths").tolist()
    responses = [[_ints(0, VOCAB, (lens[i][j],), seed, "response", i, j).tolist() for j in range(k)] for i in range(n)]
    # right or wrong answers, at least one of either kind in a group
    rewards = _ints(0, 2, (n, k), seed, "rewards")
    rewards[:, 0], rewards[:, 1] = 0, 1
    return prompts, responses, rewards.float().tolist()


# ---- what a program has in hand before the call -------------------------------------------------------------------------
def _train_engine(case, seed):
    from b200fw.train import TrainConfig, TrainEngine
    gc.collect()
    lora = case["path"] == "lora"
    grpo = case["path"] == "grpo"
    seq = case["prompt"] + case["response"] if grpo else case["seq"]
    eng = TrainEngine(TrainConfig(
        model_preset=case["model"], max_seq_len=max(64, seq), lora_rank=LORA_RANK if lora else 0, lora_alpha=LORA_ALPHA, learning_rate=LR,
        weight_decay=WD, gradient_accumulation_steps=case.get("accum", 1), grpo_beta=KL_BETA if grpo else 0.0,
        grpo_clip_eps=CLIP_EPS, max_grad_norm=CLIP, warmup_steps=0, cuda_graph_step=not grpo)).initialize()
    if not grpo:        # an engine that has trained on this shape already: its micro-steps are captured
        for _ in range(3):
            for p, r in _sft_batches(case, -1):
                eng.sft_step(p, r)
    with torch.no_grad():
        have = dict(eng.model.named_parameters())
        for name, shape in _dense_shapes(case["model"]).items():
            inside = name if name in have else name.replace("_proj.weight", "_proj.base.weight")      # under LoRA
            have[inside].copy_(_dense_weight(name, shape, seed))
        if lora:
            for (i, n), (fused, _, fan_in, fan_out) in _adapter_shapes(case["model"]).items():
                part = "mlp" if fused in ("gate_up_proj", "down_proj") else "self_attn"
                a = getattr(getattr(eng.model.layers[i], part), fused).adapters[n]
                a.lora_A.copy_(_adapter(i, n, "A", (LORA_RANK, fan_in), seed))
                a.lora_B.copy_(_adapter(i, n, "B", (fan_out, LORA_RANK), seed))
        if grpo:        # the policy has moved a little from the reference
            ref = dict(eng.ref_model.named_parameters())
            for name in _dense_shapes(case["model"]):
                ref[name].copy_(_reference_weight(name, have[name], seed))
        # ... and that takes up another run's state: its weights, no steps yet
        opt = eng.optimizer
        opt.refresh_masters_from_params()
        opt.exp_avg.zero_()
        opt.exp_avg_sq.zero_()
        opt.step_count = 0
    return eng


def _reference_weight(name, w, seed):
    """The reference differs a little everywhere, and gives random tokens less (larger logits): the KL term stays above its clamp at 0."""
    if w.dim() == 1:
        return (w.float() * 1.2).to(torch.bfloat16) if name == "norm.weight" else w
    return (w.float() * (1.0 + _normal(tuple(w.shape), 0.02, seed, "reference", name))).to(torch.bfloat16)


def _infer_engine(case, seed, lengths, decode):
    from b200fw.infer import InferenceConfig, InferenceEngine
    from b200fw.model.registry import PRESETS, build_model
    model = build_model(PRESETS[case["model"]], dtype=torch.bfloat16, device=torch.device("cuda"))
    with torch.no_grad():
        if case["model"] in DENSE:
            for name, p in model.named_parameters():
                p.requires_grad_(False).copy_(_dense_weight(name, tuple(p.shape), seed))
        else:
            for name, slot in model.checkpoint().items():
                slot.load(_sotazen_weight(name, tuple(slot.shape), seed))
    blocks = sum(-(-n // 16) + 1 for n in lengths) + 8
    return InferenceEngine(InferenceConfig.from_model_config(
        PRESETS[case["model"]], num_blocks=blocks, inference_mode="kv_cache", max_num_sequences=max(1, len(lengths)),
        kv_cache_dtype=case.get("kv", "fp16"), enable_cuda_graph=decode, seed=0), model).initialize()


def _fill_cache(case, seed, eng, lengths):
    """Pages of sequences whose newest token is still to be computed: keys as after their norm, values as projected."""
    h, layers, _, kv, _ = DENSE[case["model"]]
    for i, n in enumerate(lengths):
        eng.kv.allocate_for_sequence(i, n)
    rows = [torch.tensor(eng.kv.get_block_table(i), device="cuda")[:, None] * 16 + torch.arange(16, device="cuda")
            for i in range(len(lengths))]
    rows = torch.cat([r.reshape(-1)[:n] for r, n in zip(rows, lengths)])
    for li in range(layers):
        for pages, scales, t in zip(eng.pool.layer_kv(li), eng.pool.layer_scales(li), _cached(case, seed, li, int(rows.numel()))):
            if scales is not None:
                scales.fill_(FP8_SCALE)
                t = (t.float() / FP8_SCALE).to(torch.float8_e4m3fn).view(torch.uint8)
            pages.view(-1, kv, HEAD)[rows] = t


FP8_SCALE = 1.0 / 64


def _cached(case, seed, layer, tokens):
    h, _, _, kv, _ = DENSE[case["model"]]
    return (_normal((tokens, kv, HEAD), 1.0, seed, "k", layer).to(torch.bfloat16),
            _normal((tokens, kv, HEAD), 0.02 * h ** 0.5, seed, "v", layer).to(torch.bfloat16))


def prepare(case, seed):
    path = case["path"]
    if path in ("sft", "lora"):
        return {"path": path, "engine": _train_engine(case, seed), "batches": _sft_batches(case, seed)}
    if path == "grpo":
        return {"path": path, "engine": _train_engine(case, seed), "batch": _grpo_batch(case, seed)}
    prompts = _prompts(case, seed)
    lengths = [len(p) for p in prompts]
    eng = _infer_engine(case, seed, lengths, path == "decode")
    if path == "prefill":
        return {"path": path, "engine": eng, "prompts": prompts, "chunk": case["chunk"]}
    # decode: all but the newest token of every sequence is in the cache
    if case["model"] in DENSE:
        _fill_cache(case, seed, eng, lengths)
    else:
        for some in _chunks(prompts, 8192):
            eng.feed([(i, p[a:b]) for i, p, a, b in some], want={})
    from b200fw.infer import CUDAGraphRunner, InferenceContext
    runner, size, width = eng.runner, CUDAGraphRunner(len(lengths)).padded_size(len(lengths)), 64
    while width * 16 < max(lengths) + 1:
        width *= 2
    hybrid = hasattr(runner, "graph_inputs")

    def inputs(n):
        if hybrid:
            return runner.graph_inputs(n, width)
        i32 = dict(dtype=torch.int32, device="cuda")
        return {"tokens": torch.zeros(n, dtype=torch.long, device="cuda"), "positions": torch.zeros(n, **i32),
                "block_tables": torch.full((n, width), -1, **i32), "context_lens": torch.zeros(n, **i32),
                "segments": torch.tensor([[-1, 0, 0, 0]] * n, **i32), "slots": torch.full((n,), -1, **i32)}

    def step(t):
        if hybrid:
            return runner.forward(t["tokens"], runner.graph_context(t, width))
        ctx = InferenceContext(False, t["tokens"].shape[0], t["block_tables"], t["context_lens"], width * 16, t["segments"],
                               positions=t["positions"], slot_mapping=t["slots"])
        return runner.forward(t["tokens"], ctx, split_plan=(0, 1))
    graphs = CUDAGraphRunner(len(lengths))
    graphs.capture(size, inputs, step)
    tokens = torch.zeros(size, dtype=torch.long, device="cuda")
    tokens[:len(lengths)] = torch.tensor([p[-1] for p in prompts], device="cuda")
    return {"path": path, "engine": eng, "graphs": graphs, "size": size, "width": width, "hybrid": hybrid, "tokens": tokens,
            "ids": list(range(len(lengths)))}


def _chunks(prompts, budget):
    """Steps of at most about ``budget`` tokens: lists of (sequence, prompt, from, to)."""
    step, room = [], budget
    for i, p in enumerate(prompts):
        at = 0
        while at < len(p):
            n = min(room, len(p) - at)
            step.append((i, p, at, at + n))
            at, room = at + n, room - n
            if room == 0:
                yield step
                step, room = [], budget
    if step:
        yield step


# ---- one pass -----------------------------------------------------------------------------------------------------------
def run(state):
    eng = state["engine"]
    if state["path"] in ("sft", "lora", "grpo"):
        if state["path"] == "grpo":
            losses = [eng.grpo_step(*state["batch"])]
        else:
            losses = [eng.sft_step(p, r) for p, r in state["batches"]]
        opt = eng.optimizer
        # GRPO: the two parts of the loss (their sum may lie near zero)
        parts = [losses[0].policy_loss, losses[0].kl_divergence] if state["path"] == "grpo" else [m.loss for m in losses]
        return {"loss": parts, "grad_norm": losses[-1].grad_norm, "weights": opt.master, "momentum": opt.exp_avg,
                "variance": opt.exp_avg_sq}
    if state["path"] == "prefill":
        out = {}
        for some in _chunks(state["prompts"], state["chunk"]):
            last = {i: [b - a - 1] for i, p, a, b in some if b == len(p)}
            got = eng.feed([(i, p[a:b]) for i, p, a, b in some], want=last)
            out.update({i: got[i] for i in last})
        for i in out:
            eng.release(i)
        return out
    runner, g, size = eng.runner, state["graphs"], state["size"]
    ctx = runner.prepare_decode(state["ids"], pad_to=size, max_blocks=state["width"])
    if state["hybrid"]:
        values = runner.graph_values(ctx)
    else:
        values = {"positions": ctx.positions, "block_tables": ctx.block_tables, "context_lens": ctx.context_lens,
                  "segments": ctx.store_segments, "slots": ctx.slot_mapping}
    return g.replay(size, {"tokens": state["tokens"], **values})[:len(state["ids"])]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def work(case):
    path, model = case["path"], case["model"]
    if model in SOTAZEN:
        c = SOTAZEN[model]
        W, H, D = c["width"], c["heads"], HEAD
        mix = {"lightning": 5 * W * H * D, "differential": W * D * (2 * H + 3 * c["kv_heads"] + 2 * H),
               "latent": W * (H * (D + c["rot"]) + c["rank"] + c["rot"] + H * D) + 2 * c["rank"] * H * D}
        body = sum(mix[k] + 2 * W * c["ff"] for _, k in _sotazen_layers(model))
        hidden, heads, layers = W, H, c["depth"]
    else:
        hidden, layers, heads, kv, ff = DENSE[model]
        body = layers * (hidden * HEAD * 2 * (heads + kv) + 3 * hidden * ff)
    head = VOCAB * hidden
    if path in ("sft", "lora", "grpo"):
        if path == "grpo":
            # samples are 5/8 of the longest response on average
            rows = [(case["prompt"] + case["response"] * 0.625, case["response"] * 0.625)] * (case["prompts"] * case["samples"])
        else:
            rows = [(case["seq"], case["seq"] - case["seq"] // 2)] * (case["batch"] * case["accum"])
        att = sum(2.0 * s * s * HEAD * heads * layers for s, _ in rows)
        fwd = 2.0 * body * sum(s for s, _ in rows) + 2.0 * head * sum(r for _, r in rows) + att
        if path == "lora":
            adapters = sum(LORA_RANK * (a + b) for _, _, a, b in _adapter_shapes(model).values())
            return {"bytes": 2.0 * (body + head) + 24.0 * adapters, "flops": 2 * fwd + 1.5 * att + 6.0 * adapters * sum(s for s, _ in rows)}
        # master weights and both moments in and out, 16-bit weights in and out (and the reference's in)
        return {"bytes": (body + head) * (28.0 + (2.0 if path == "grpo" else 0.0)), "flops": 3 * fwd + 0.5 * att + (fwd if path == "grpo" else 0.0)}
    n = case["batch"]
    L = case["seq"] if path == "prefill" else case["context"]
    L = L if n == 1 else 0.75 * L
    if path == "prefill":
        pairs = 2.0 * L * L * HEAD * heads
        if model in SOTAZEN:
            c, w = SOTAZEN[model], min(L, SOTAZEN[model]["window"])
            pairs = sum({"latent": 0.5 * pairs * (2 + c["rot"] / HEAD), "differential": 2 * 4.0 * (L * w - 0.5 * w * w) * HEAD * heads,
                         "lightning": 4.0 * L * HEAD * HEAD * heads}[k] for _, k in _sotazen_layers(model))
        else:
            pairs *= layers
        return {"bytes": 2.0 * (body + head) + n * VOCAB * (4.0 if model in SOTAZEN else 2.0), "flops": 2.0 * body * n * L + 2.0 * head * n + n * pairs}
    if model in SOTAZEN:
        c, w = SOTAZEN[model], min(L, SOTAZEN[model]["window"])
        cache = sum({"latent": 2.0 * L * (c["rank"] + c["rot"]), "differential": 2.0 * w * 3 * HEAD * c["kv_heads"],
                     "lightning": 8.0 * HEAD * HEAD * heads}[k] for _, k in _sotazen_layers(model))
        flops = sum({"latent": 2.0 * L * heads * (2 * c["rank"] + c["rot"]), "differential": 2 * 4.0 * w * heads * HEAD,
                     "lightning": 4.0 * HEAD * HEAD * heads}[k] for _, k in _sotazen_layers(model))
    else:
        cache = layers * L * kv * HEAD * 2 * (1.0 if case["kv"] == "fp8" else 2.0)
        flops = layers * 4.0 * L * heads * HEAD
    return {"bytes": 2.0 * (body + head) + n * (cache + VOCAB * (4.0 if model in SOTAZEN else 2.0)),
            "flops": n * (2.0 * (body + head) + flops)}


def tolerance(case):
    # a bf16 residual stream of 28 to 36 layers: two orders of summation differ by up to 1.5e-2 in logits and in gradients
    return {"rel": 0.03}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------
def _rms(x, w=None):
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)
    return x if w is None else x * w


def _rope_half(x, pos):
    """Rotary positions for ``x [.., T, heads, 128]``: channel i turns with channel i + 64."""
    f = THETA ** (-torch.arange(0, HEAD, 2, device="cuda", dtype=torch.float64) / HEAD)
    a = pos.double()[:, None] * f
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = x[..., :HEAD // 2], x[..., HEAD // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _rope_pairs(x, pos, base):
    """``x [T, heads, dims]``: channels 2 i and 2 i + 1 turn together."""
    d = x.shape[-1]
    a = pos.double()[:, None] * base ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).reshape(x.shape)


def _causal(q, k, v):
    """``q [T, H, d]``, ``k, v [T, G, d]``: causal softmax attention, a block of queries at a time."""
    T, H, d = q.shape
    g = H // k.shape[1]
    kh, vh, out = k.repeat_interleave(g, 1).transpose(0, 1), v.repeat_interleave(g, 1).transpose(0, 1), []
    for a in range(0, T, 1024):
        b = min(T, a + 1024)
        s = q[a:b].transpose(0, 1) @ kh[:, :b].transpose(1, 2) * d ** -0.5
        s = s.masked_fill(torch.arange(b, device="cuda") > torch.arange(a, b, device="cuda")[:, None], -math.inf)
        out.append((torch.softmax(s, -1) @ vh[:, :b]).transpose(0, 1))
    return torch.cat(out)


class _Lora:
    """Fused projections with their adapters, for the 64-bit model."""

    def __init__(self, case, params):
        self.params, self.parts = params, {}
        for (i, n), (fused, rows, _, _) in _adapter_shapes(case["model"]).items():
            self.parts.setdefault((i, fused), []).append(((i, n), rows))

    def __call__(self, i, fused, x, y):
        add = [x @ self.params[key + ("A",)].T @ self.params[key + ("B",)].T * (LORA_ALPHA / LORA_RANK) for key, _ in self.parts[(i, fused)]]
        return y + torch.cat(add, -1)


def _dense_layer(case, i, x, rows, w, lora=None):
    """One layer over packed sequences ``x [T, hidden]``; ``rows``: their (first, last + 1)."""
    h, _, heads, kv, ff = DENSE[case["model"]]
    p = f"layers.{i}."

    def lin(part, fused, t):
        y = t @ w(p + f"{part}.{fused}.weight").T
        return y if lora is None else lora(i, fused, t, y)
    n = _rms(x, w(p + "input_layernorm.weight"))
    q, k, v = lin("self_attn", "qkv_proj", n).reshape(-1, heads + 2 * kv, HEAD).split([heads, kv, kv], 1)
    q, k = _rms(q, w(p + "self_attn.q_norm.weight")), _rms(k, w(p + "self_attn.k_norm.weight"))
    att = []
    for a, b in rows:
        pos = torch.arange(b - a, device="cuda")
        att.append(_causal(_rope_half(q[a:b], pos), _rope_half(k[a:b], pos), v[a:b]))
    x = x + lin("self_attn", "o_proj", torch.cat(att).reshape(x.shape[0], -1))
    n = _rms(x, w(p + "post_attention_layernorm.weight"))
    gate, up = lin("mlp", "gate_up_proj", n).split(ff, -1)
    return x + lin("mlp", "down_proj", F.silu(gate) * up)


def _hidden(case, ids, rows, w, lora=None, grad=False):
    """Final normed hidden states of packed sequences."""
    x = w("embed_tokens")[ids]
    for i in range(DENSE[case["model"]][1]):
        if grad:
            x = checkpoint(lambda t, i=i: _dense_layer(case, i, t, rows, w, lora), x, use_reentrant=False)
        else:
            x = _dense_layer(case, i, x, rows, w, lora)
    return _rms(x, w("norm.weight"))


def _logprobs(h, table, labels):
    """Log-probability of each row's label, 1024 rows at a time."""
    def some(a, t, l):
        return torch.log_softmax(a @ t.T, -1).gather(-1, l[:, None])[:, 0]
    return torch.cat([checkpoint(some, h[a:a + 1024], table, labels[a:a + 1024], use_reentrant=False) for a in range(0, h.shape[0], 1024)])


def _pack(rows):
    at, spans = 0, []
    for r in rows:
        spans.append((at, at + len(r)))
        at += len(r)
    return torch.tensor([t for r in rows for t in r], device="cuda"), spans


def _scored(spans, prompts):
    """Rows whose next token is part of a response."""
    return torch.cat([torch.arange(a + n - 1, b - 1, device="cuda") for (a, b), n in zip(spans, prompts)])


def _exact_training(case, seed):
    shapes, lora = _dense_shapes(case["model"]), None
    start = {n: _dense_weight(n, s, seed).double() for n, s in shapes.items()}
    if case["path"] == "lora":
        train = {}
        for (i, n), (_, _, fan_in, fan_out) in _adapter_shapes(case["model"]).items():
            train[(i, n, "A")] = _adapter(i, n, "A", (LORA_RANK, fan_in), seed).double()
            train[(i, n, "B")] = _adapter(i, n, "B", (fan_out, LORA_RANK), seed).double()
        lora = _Lora(case, train)
    else:
        train = start
    for t in train.values():
        t.requires_grad_(True)
    w, losses = start.__getitem__, []
    if case["path"] == "grpo":
        prompts, groups, rewards = _grpo_batch(case, seed)
        ids, spans = _pack([p + r for p, g in zip(prompts, groups) for r in g])
        rows = _scored(spans, [case["prompt"]] * len(spans))
        adv = []
        for r in rewards:
            t = torch.tensor(r, dtype=torch.float64)
            adv += ((t - t.mean()) / (t.std(unbiased=False) + 1e-8)).tolist()
        adv = torch.cat([torch.full((b - a - case["prompt"],), v, dtype=torch.float64, device="cuda") for (a, b), v in zip(spans, adv)])
        with torch.no_grad():
            def ref(name):
                return _reference_weight(name, _dense_weight(name, shapes[name], seed), seed).double()
            base = _logprobs(_hidden(case, ids, spans, ref)[rows], ref("embed_tokens"), ids[rows + 1])
        lp = _logprobs(_hidden(case, ids, spans, w, grad=True)[rows], w("embed_tokens"), ids[rows + 1])
        ratio = torch.exp(lp - lp.detach())
        policy = -torch.minimum(ratio * adv, ratio.clamp(1 - CLIP_EPS, 1 + CLIP_EPS) * adv).sum() / lp.numel()
        kl = ((lp - base).sum() / lp.numel()).clamp(min=0.0)
        (policy + KL_BETA * kl).backward()
        losses += [float(policy), float(kl)]
    else:
        for prompts, responses in _sft_batches(case, seed):
            ids, spans = _pack([p + r for p, r in zip(prompts, responses)])
            rows = _scored(spans, [len(p) for p in prompts])
            loss = -_logprobs(_hidden(case, ids, spans, w, lora, grad=True)[rows], w("embed_tokens"), ids[rows + 1]).mean()
            (loss / case["accum"]).backward()
            losses.append(float(loss))
    with torch.no_grad():
        order = list(train.values())[::-1]          # the optimizer keeps its parameters back to front
        g = torch.cat([t.grad.reshape(-1) for t in order])
        norm = float(g.norm())
        g *= min(1.0, CLIP / (norm + 1e-6))
        p = torch.cat([t.reshape(-1) for t in order])
        m, v = (1 - BETA1) * g, (1 - BETA2) * g * g
        p = p * (1 - LR * WD) - LR * g / (g.abs() + ADAM_EPS)
    # losses and norm are single numbers, whose distance from these is chance: they are compared, not measured
    return {"loss": [None] * len(losses), "grad_norm": None, "weights": p, "momentum": m, "variance": v}


def _lazy(case, seed):
    shapes = _dense_shapes(case["model"])
    return lambda name: _dense_weight(name, shapes[name], seed).double()


def _exact_decode(case, seed):
    h, layers, heads, kv, ff = DENSE[case["model"]]
    w, prompts = _lazy(case, seed), _prompts(case, seed)
    lengths = [len(p) for p in prompts]
    pos = torch.tensor(lengths, device="cuda") - 1
    x = w("embed_tokens")[torch.tensor([p[-1] for p in prompts], device="cuda")]
    for i in range(layers):
        p = f"layers.{i}."
        q, k, v = (_rms(x, w(p + "input_layernorm.weight")) @ w(p + "self_attn.qkv_proj.weight").T).reshape(
            -1, heads + 2 * kv, HEAD).split([heads, kv, kv], 1)
        q = _rope_half(_rms(q, w(p + "self_attn.q_norm.weight")), pos)
        k = _rope_half(_rms(k, w(p + "self_attn.k_norm.weight")), pos)
        ck, cv = _cached(case, seed, i, sum(lengths))
        if case["kv"] == "fp8":
            ck, cv = ((t.float() / FP8_SCALE).to(torch.float8_e4m3fn).float() * FP8_SCALE for t in (ck, cv))
        att, at = [], 0
        for b, n in enumerate(lengths):
            kb = torch.cat([ck[at:at + n - 1].double(), k[b:b + 1]]).transpose(0, 1)        # [kv, n, 128]
            vb = torch.cat([cv[at:at + n - 1].double(), v[b:b + 1]]).transpose(0, 1)
            s = torch.softmax(q[b].reshape(kv, -1, HEAD) @ kb.transpose(1, 2) * HEAD ** -0.5, -1)
            att.append((s @ vb).reshape(-1))
            at += n
        x = x + torch.stack(att) @ w(p + "self_attn.o_proj.weight").T
        gate, up = (_rms(x, w(p + "post_attention_layernorm.weight")) @ w(p + "mlp.gate_up_proj.weight").T).split(ff, -1)
        x = x + (F.silu(gate) * up) @ w(p + "mlp.down_proj.weight").T
    return _rms(x, w("norm.weight")) @ w("embed_tokens").T


def _softmax_rows(q, k, v, scale, window=0, cap=0.0, sink=None):
    """``q, k [H, T, d]``, ``v [H, T, e]``: causal, perhaps in a window, scores pressed through cap tanh(s / cap), an extra term
    exp(sink) in the denominator."""
    T, out = q.shape[1], []
    for a in range(0, T, 512):
        b = min(T, a + 512)
        s = q[:, a:b] @ k[:, :b].transpose(1, 2) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        far = torch.arange(a, b, device="cuda")[:, None] - torch.arange(b, device="cuda")
        s = s.masked_fill((far < 0) | ((far >= window) if window else (far < 0)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, b - a, 1)], -1)
        out.append(torch.softmax(s, -1)[..., :b] @ v[:, :b])
    return torch.cat(out, 1)


def _lightning(q, k, v, decay):
    """``[H, T, d]``: sums of v with the product of q and k, decaying with the distance."""
    T, out, d = q.shape[1], [], torch.log(decay)[:, None, None]
    for a in range(0, T, 512):
        b = min(T, a + 512)
        far = (torch.arange(a, b, device="cuda")[:, None] - torch.arange(b, device="cuda")).double()
        out.append((q[:, a:b] @ k[:, :b].transpose(1, 2) * torch.exp(d * far.clamp(min=0)) * (far >= 0)) @ v[:, :b])
    return torch.cat(out, 1)


def _exact_sotazen(case, seed):
    c = SOTAZEN[case["model"]]
    W, H, G, D, R, C = c["width"], c["heads"], c["kv_heads"], HEAD, c["rot"], c["rank"]
    ids, spans = _pack(_prompts(case, seed))

    def w(name, *shape):
        return _sotazen_weight(name, shape, seed).double()

    def heads(t, n):
        return t.reshape(t.shape[0], n, -1)
    alpha, emb = (2.0 * c["depth"]) ** 0.25, w("embed", VOCAB, W)
    x = emb[ids] * W ** 0.5
    for i, kind in _sotazen_layers(case["model"]):
        p = f"l{i}.mix."
        if kind == "lightning":
            q, k, v = (heads(F.silu(x @ w(p + n, H * D, W).T), H) for n in "qkv")
            decay = 1.0 - 2.0 ** (-5.0 - 7.0 * torch.arange(H, device="cuda", dtype=torch.float64) / max(1, H - 1))
            o = torch.cat([_lightning(*(t[a:b].transpose(0, 1) for t in (q, k, v)), decay).transpose(0, 1) for a, b in spans])
            o = _rms(o.reshape(-1, H * D), w(p + "norm", H * D)) * torch.sigmoid(x @ w(p + "g", H * D, W).T)
            y = o @ w(p + "o", W, H * D).T
        elif kind == "differential":
            q, k, v = (heads(x @ w(p + n, r * D, W).T + w(p + n + ".b", r * D), r) for n, r in (("q", 2 * H), ("k", 2 * G), ("v", G)))
            q, k = _rms(q, w(p + "q.norm", D)), _rms(k, w(p + "k.norm", D))
            lam = torch.exp((w(p + "lq1", D) * w(p + "lk1", D)).sum()) - torch.exp((w(p + "lq2", D) * w(p + "lk2", D)).sum()) + 0.4
            outs = []
            for a, b in spans:
                pos = torch.arange(b - a, device="cuda")
                qs = _rope_pairs(q[a:b], pos, 10000.0).transpose(0, 1)
                ks = _rope_pairs(k[a:b], pos, 10000.0).reshape(b - a, G, 2, D).repeat_interleave(H // G, 1).reshape(b - a, 2 * H, D)
                vs = v[a:b].repeat_interleave(H // G, 1).repeat_interleave(2, 1)
                o = _softmax_rows(qs, ks.transpose(0, 1), vs.transpose(0, 1), D ** -0.5, c["window"], 30.0)
                outs.append((o[0::2] - lam * o[1::2]).transpose(0, 1))
            o = (_rms(torch.cat(outs)) * 0.6).reshape(-1, H * D) * torch.sigmoid(x @ w(p + "g", H * D, W).T)
            y = o @ w(p + "o", W, H * D).T + w(p + "o.b", W)
        else:
            q = heads(x @ w(p + "q", H * (D + R), W).T, H)
            down = x @ w(p + "dkv", C + R, W).T
            lat = _rms(down[:, :C], w(p + "dkv.norm", C))
            k, v = heads(lat @ w(p + "uk", H * D, C).T, H), heads(lat @ w(p + "uv", H * D, C).T, H)
            outs = []
            for a, b in spans:
                pos = torch.arange(b - a, device="cuda")
                kr = _rope_pairs(down[a:b, None, C:], pos, 10000.0).expand(-1, H, -1)
                qs = torch.cat([q[a:b, :, :D], _rope_pairs(q[a:b, :, D:], pos, 10000.0)], -1)
                o = _softmax_rows(qs.transpose(0, 1), torch.cat([k[a:b], kr], -1).transpose(0, 1), v[a:b].transpose(0, 1), (D + R) ** -0.5,
                                  sink=w(p + "sink", H))
                outs.append(o.transpose(0, 1))
            y = torch.cat(outs).reshape(-1, H * D) @ w(p + "o", W, H * D).T
        x = _rms(alpha * x + y, w(f"l{i}.norm1", W))
        y = torch.clamp(x @ w(f"l{i}.mlp.up", c["ff"], W).T, min=0.0) ** 2 @ w(f"l{i}.mlp.down", W, c["ff"]).T
        x = _rms(alpha * x + y, w(f"l{i}.norm2", W))
    last = torch.tensor([b - 1 for _, b in spans], device="cuda")
    return _rms(x[last], w("final.norm", W)) @ emb.T


def exact(case, seed):
    if case["path"] in ("sft", "lora", "grpo"):
        return _exact_training(case, seed)
    with torch.no_grad():
        if case["model"] in SOTAZEN:
            out = _exact_sotazen(case, seed)
        elif case["path"] == "decode":
            return _exact_decode(case, seed)
        else:
            ids, spans = _pack(_prompts(case, seed))
            w = _lazy(case, seed)
            h = _hidden(case, ids, spans, w)[torch.tensor([b - 1 for _, b in spans], device="cuda")]
            out = h @ w("embed_tokens").T
        return out if case["path"] == "decode" else {i: out[i:i + 1] for i in range(case["batch"])}
