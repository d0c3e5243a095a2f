"""Performance cases: what the main phases of a reinforcement-learning run ask of this framework.

A GRPO iteration generates responses (prefill, then one decode step per token), recomputes log-probabilities with the
trainer's weights, and runs forward and backward over packed micro-batches. Each kind of case below is one of those calls
through the public model and op entry points, at the widths of the model presets (with fewer layers where a pass over all
of them would only repeat the same work) and at sequence lengths of the benchmark configurations: prompts of 128 to 512
tokens with responses up to 4096 (Qwen3-1.7B), up to 16384 (Qwen3-8B) and up to 8192 (Qwen3-30B-A3B, Qwen2.5-7B in fp8).

* ``trunk_train``: decoder blocks and final norm of a packed micro-batch, forward and backward into fp32 main gradients.
* ``head_train``: LM head, log-probabilities, entropy, decoupled PPO loss and the backward pass of all of it.
* ``logp``: embedding, decoder blocks, log-probabilities and entropy of a micro-batch, without gradients.
* ``prefill``: prompts through all layers into the paged cache, then the first token of every response.
* ``decode``: one token for every running sequence, as the captured graph that the rollout engine replays.
* ``sample``: top-p / top-k sampling from materialised logits (requests that filter, and every first token).
"""

from __future__ import annotations

import dataclasses
import math
import random

import torch
import torch.nn.functional as F

PAGE = 16
HEAD = 128
EPS = 1e-6
THETA = 1e6

# hidden, layers, query heads, key / value heads, feed-forward width, vocabulary, q/k norm, experts, experts per token, expert width
WIDTHS = {
    "qwen3-1.7b": dict(H=2048, L=28, Hq=16, Hkv=8, I=6144, V=151936, norm=True, E=0, k=0, Ie=0),
    "qwen3-8b": dict(H=4096, L=36, Hq=32, Hkv=8, I=12288, V=151936, norm=True, E=0, k=0, Ie=0),
    "qwen2.5-7b": dict(H=3584, L=28, Hq=28, Hkv=4, I=18944, V=152064, norm=False, E=0, k=0, Ie=0),
    "qwen3-30b-a3b": dict(H=2048, L=48, Hq=32, Hkv=4, I=0, V=151936, norm=True, E=128, k=8, Ie=768),
}


def listed():
    return [
        # a short micro-batch: small prompts and answers, or the remainder of a batch; bound by launches and small grids
        dict(name="train_short_1.7b", kind="trunk_train", model="qwen3-1.7b", layers=2, tokens=900, shortest=40, longest=320, fp8=False, lens=1),
        # the benchmark's own micro-batch: prompts and responses up to 4608 tokens packed to 16384
        dict(name="train_packed_1.7b", kind="trunk_train", model="qwen3-1.7b", layers=4, tokens=16384, shortest=384, longest=4608, fp8=False, lens=2),
        # long reasoning traces: attention is most of the work
        dict(name="train_long_8b", kind="trunk_train", model="qwen3-8b", layers=2, tokens=32768, shortest=1536, longest=16896, fp8=False, lens=3),
        # mixture of experts: routing, grouped products, scatter and combine
        dict(name="train_moe_30b", kind="trunk_train", model="qwen3-30b-a3b", layers=2, tokens=12000, shortest=1024, longest=8704, fp8=False, lens=4),
        # block-scaled fp8 forward products, projections with bias, seven query heads to a key head
        dict(name="train_fp8_7b", kind="trunk_train", model="qwen2.5-7b", layers=1, tokens=8192, shortest=512, longest=8192, fp8=True, lens=5),
        # the loss end of a training step: vocabulary-sized products around the PPO loss
        dict(name="head_train_1.7b", kind="head_train", model="qwen3-1.7b", tokens=8192),
        # log-probabilities recomputed by the trainer before the update
        dict(name="logp_1.7b", kind="logp", model="qwen3-1.7b", layers=4, tokens=16384, shortest=384, longest=4608, lens=6),
        # a scheduler step that admits the prompts of one group batch
        dict(name="prefill_1.7b", kind="prefill", model="qwen3-1.7b", layers=28, tokens=2600, shortest=128, longest=512, lens=7),
        # the straggler of a batch, or an interactive request: one sequence
        dict(name="decode_1_1.7b", kind="decode", model="qwen3-1.7b", layers=28, batch=1, shortest=700, longest=1400, context=4608, lens=8),
        # the tail of a batch of long traces
        dict(name="decode_16_8b", kind="decode", model="qwen3-8b", layers=12, batch=16, shortest=1024, longest=8192, context=16896, lens=9),
        # a full rollout batch
        dict(name="decode_256_1.7b", kind="decode", model="qwen3-1.7b", layers=28, batch=256, shortest=300, longest=2000, context=4608, lens=10),
        # a batch of requests with nucleus sampling
        dict(name="sample_top_p_128", kind="sample", batch=128, vocab=151936, top_p=0.95, top_k=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above. The ranges overlap the listed cases; sizes are seldom round."""
    kind = rng.choice(["trunk_train"] * 5 + ["head_train", "logp", "prefill"] + ["decode"] * 3 + ["sample"])
    lens = rng.randrange(1 << 20)
    if kind == "trunk_train":
        model, layers, most = rng.choice([("qwen3-1.7b", 4, 16384), ("qwen3-1.7b", 2, 32768), ("qwen3-8b", 2, 24000),
                                          ("qwen3-30b-a3b", 2, 12000), ("qwen2.5-7b", 1, 12000)])
        tokens = _log(rng, 600, most)
        longest = min(tokens, _log(rng, 256, 16896))
        return dict(kind=kind, model=model, layers=rng.randint(1, layers), tokens=tokens, shortest=max(1, longest // rng.randint(2, 12)),
                    longest=longest, fp8=model == "qwen2.5-7b" and rng.random() < 0.7, lens=lens)
    if kind == "head_train":
        return dict(kind=kind, model=rng.choice(["qwen3-1.7b", "qwen2.5-7b"]), tokens=_log(rng, 500, 8192))
    if kind == "logp":
        tokens = _log(rng, 600, 16384)
        longest = min(tokens, _log(rng, 256, 8704))
        return dict(kind=kind, model="qwen3-1.7b", layers=rng.randint(1, 4), tokens=tokens, shortest=max(1, longest // rng.randint(2, 12)),
                    longest=longest, lens=lens)
    if kind == "prefill":
        tokens = _log(rng, 130, 8192)
        return dict(kind=kind, model="qwen3-1.7b", layers=rng.randint(7, 28), tokens=tokens, shortest=min(tokens, rng.randint(16, 256)),
                    longest=min(tokens, _log(rng, 257, 4096)), lens=lens)
    if kind == "decode":
        model = rng.choice(["qwen3-1.7b", "qwen3-1.7b", "qwen3-8b"])
        big = model == "qwen3-8b"
        batch = _log(rng, 1, 24 if big else 256)
        longest = min(_log(rng, 64, 16384), (131072 if big else 524288) // batch)
        return dict(kind=kind, model=model, layers=rng.randint(4, 12) if big else rng.randint(7, 28), batch=batch,
                    shortest=max(1, longest // rng.randint(2, 8)), longest=longest, context=max(longest, _log(rng, 1024, 16896)), lens=lens)
    return dict(kind=kind, batch=_log(rng, 1, 256), vocab=rng.choice([151936, 152064, 128256, 32000]), top_p=rng.choice([0.8, 0.9, 0.95, 1.0]),
                top_k=rng.choice([0, 0, 20, 50]))


# ------------------------------------------------------------------------------------------------- inputs


def _lengths(case):
    """Lengths of the packed sequences, from the case alone: the last one is what is left of the micro-batch."""
    r, left, out = random.Random(case["lens"]), case["tokens"], []
    while left:
        n = min(left, r.randint(case["shortest"], case["longest"]))
        out.append(n)
        left -= n
    return out


def _contexts(case):
    r = random.Random(case["lens"])
    return [r.randint(case["shortest"], case["longest"]) for _ in range(case["batch"])]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=g)


def _weights(case, g, vocab, layers):
    """Random weights at trained magnitudes: projections of 0.02, the ones that write the residual stream scaled down
    with depth, norm weights around one, and routers sharp enough that the choice of experts does not hang on rounding."""
    m = WIDTHS[case["model"]]
    H, q, kv = m["H"], m["Hq"] * HEAD, m["Hkv"] * HEAD
    w, out = {}, 0.02 / math.sqrt(2 * max(layers, 2))
    for i in range(layers):
        p = f"layers.{i}."
        w[p + "input_norm"] = _normal(g, H, std=0.1, mean=1.0)
        w[p + "attn.qkv"] = _normal(g, q + 2 * kv, H, std=0.02)
        if not m["norm"]:
            w[p + "attn.qkv_bias"] = _normal(g, q + 2 * kv, std=0.1)
        w[p + "attn.o"] = _normal(g, H, q, std=out)
        if m["norm"]:
            w[p + "attn.q_norm"] = _normal(g, HEAD, std=0.1, mean=1.0)
            w[p + "attn.k_norm"] = _normal(g, HEAD, std=0.1, mean=1.0)
        w[p + "post_norm"] = _normal(g, H, std=0.1, mean=1.0)
        if m["E"]:
            w[p + "mlp.router"] = _normal(g, m["E"], H, std=0.1)
            w[p + "mlp.gate_up"] = _normal(g, m["E"], 2 * m["Ie"], H, std=0.02)
            w[p + "mlp.down"] = _normal(g, m["E"], H, m["Ie"], std=out)
        else:
            w[p + "mlp.gate_up"] = _normal(g, 2 * m["I"], H, std=0.02)
            w[p + "mlp.down"] = _normal(g, H, m["I"], std=out)
    w["norm"] = _normal(g, H, std=0.1, mean=1.0)
    if vocab:
        # A trained model's next-token distributions are peaked: with a head tied to the embedding and a residual stream
        # that keeps it, the token that a position already holds gets nearly all of the mass.
        std = 0.45 if H <= 2048 else 1.5  # wider feed-forwards add more to the stream
        w["embed"] = _normal(g, m["V"], H, std=std)
        w["norm"] *= 20.0 / (0.7 * H * std)
    return w


def _model(case, w, vocab):
    """The framework's model of this preset on the weights ``w``."""
    from areal_b200.models.config import PRESETS
    from areal_b200.models.qwen import QwenModel

    over = dict(num_hidden_layers=case["layers"], tie_word_embeddings=True, fp8=bool(case.get("fp8")))
    if not vocab:
        over["vocab_size"] = 128  # the blocks get embeddings as their input
    model = QwenModel(dataclasses.replace(PRESETS[case["model"]], **over), device="cuda")
    for name, p in model.named_parameters():
        if name in w:
            p.data = w[name]
    model.rope("cuda")
    return model


def _packed(case):
    from areal_b200.ops.attention import VarlenMeta

    lens = _lengths(case)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    pos = torch.cat([torch.arange(n) for n in lens]).to(device="cuda", dtype=torch.int32)
    return VarlenMeta(cu, "cuda"), pos


def _pages(case, g):
    """Block table and number of pages of a decode batch: the page that the new token goes to comes from the last
    ``batch`` pages, the others are spread over the cache as a long-running scheduler leaves them."""
    ctx, width = _contexts(case), -(-case["context"] // PAGE)
    full = [(n - 1) // PAGE for n in ctx]
    total = sum(full)
    order = torch.randperm(total, generator=torch.Generator().manual_seed(case["lens"])).tolist()
    table, at = torch.zeros((len(ctx), width), dtype=torch.int32), 0
    for b, n in enumerate(full):
        table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        table[b, n] = total + b
        at += n
    return ctx, table, total + len(ctx)


def _caches(case, g, pages):
    m = WIDTHS[case["model"]]
    shape = (case["layers"], pages, m["Hkv"], PAGE, HEAD)
    return _normal(g, *shape), _normal(g, *shape, std=0.9)


def _trunk_inputs(case, seed):
    g, H = _gen(seed), WIDTHS[case["model"]]["H"]
    w = _weights(case, g, False, case["layers"])
    x = _normal(g, case["tokens"], H)
    dy = _normal(g, case["tokens"], H, std=1e-3)
    return w, x, dy


def _head_inputs(case, seed):
    """Hidden states that lean towards their label as a trained model's do; proximal and behaviour log-probabilities close to
    what the head gives, as they are after a few updates."""
    m, g, T = WIDTHS[case["model"]], _gen(seed), case["tokens"]
    w = _normal(g, m["V"], m["H"], std=0.02)
    labels = torch.randint(0, m["V"], (T,), device="cuda", generator=g, dtype=torch.int32)
    c = torch.empty(T, 1, device="cuda").uniform_(0.2, 0.45, generator=g) * math.sqrt(2048 / m["H"])
    x = ((1 - c * c).sqrt() * _normal(g, T, m["H"], dtype=torch.float32) + c * 50 * w[labels.long()].float()).bfloat16()
    now = torch.cat([(z := (a @ w.t()).float()).gather(1, b[:, None].long())[:, 0] - z.logsumexp(1)
                     for a, b in zip(x.split(2048), labels.split(2048))])
    prox = now + 0.03 * _normal(g, T, dtype=torch.float32)
    behav = prox + 0.05 * _normal(g, T, dtype=torch.float32)
    adv = _normal(g, T, dtype=torch.float32)
    mask = torch.empty(T, device="cuda").uniform_(generator=g) < 0.85
    return dict(w=w, x=x, labels=labels, prox=prox, behav=behav, adv=adv, mask=mask)


def _token_inputs(case, seed, n):
    m, g = WIDTHS[case["model"]], _gen(seed)
    w = _weights(case, g, True, case["layers"])
    return g, w, torch.randint(0, m["V"], (n,), device="cuda", generator=g, dtype=torch.int32)


def _sample_inputs(case, seed):
    """Logits of a trained model's shape: a few dozen likely tokens over a long tail of unlikely ones."""
    g, B, V = _gen(seed), case["batch"], case["vocab"]
    x = _normal(g, B, V, std=1.5, dtype=torch.float32)
    likely = torch.randint(0, V, (B, 64), device="cuda", generator=g)
    x.scatter_(1, likely, 14 + 2.5 * _normal(g, B, 64, dtype=torch.float32))
    temp = torch.empty(B, device="cuda").uniform_(0.6, 1.0, generator=g)
    u = torch.empty(B, device="cuda").uniform_(0.001, 0.999, generator=g)
    return x, temp, u


def _prefill_slots(lens):
    """Flat cache slots of packed prompts whose pages follow one another, and the number of pages."""
    out, page = [], 0
    for n in lens:
        out.append(torch.arange(n) + page * PAGE)
        page += -(-n // PAGE)
    return torch.cat(out).to(device="cuda", dtype=torch.int64), page


def prepare(case, seed):
    kind, state = case["kind"], dict(kind=case["kind"])
    if kind == "trunk_train":
        w, x, dy = _trunk_inputs(case, seed)
        model = _model(case, w, False)
        meta, pos = _packed(case)
        named = [(n, p) for n, p in model.named_parameters() if n in w]
        main = torch.zeros(sum(p.numel() for _, p in named), dtype=torch.float32, device="cuda")
        at = 0
        for _, p in named:  # one fp32 buffer for all main gradients, as the training engine lays them out
            p.main_grad = main[at:at + p.numel()].view(p.shape)
            at += p.numel()
        state.update(model=model.train(), meta=meta, pos=pos, x=x.requires_grad_(), dy=dy, named=named, main=main)
    elif kind == "head_train":
        state.update(_head_inputs(case, seed))
        state["x"].requires_grad_()
        state["w"].requires_grad_()
        state["w"].main_grad = torch.zeros(state["w"].shape, dtype=torch.float32, device="cuda")
        state["count"] = float(state["mask"].sum())
    elif kind == "logp":
        _, w, ids = _token_inputs(case, seed, case["tokens"])
        meta, pos = _packed(case)
        state.update(model=_model(case, w, True).eval(), meta=meta, pos=pos, ids=ids)
    elif kind == "prefill":
        g, w, ids = _token_inputs(case, seed, case["tokens"])
        meta, pos = _packed(case)
        lens, m = _lengths(case), WIDTHS[case["model"]]
        slots, pages = _prefill_slots(lens)
        k, v = (torch.zeros((case["layers"], pages, m["Hkv"], PAGE, HEAD), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        state.update(model=_model(case, w, True).eval(), meta=meta, pos=pos, ids=ids, slots=slots, k=k, v=v,
                     caches=list(zip(k, v)), last=torch.tensor([sum(lens[:i + 1]) - 1 for i in range(len(lens))], device="cuda"),
                     temp=torch.ones(len(lens), device="cuda"), u=torch.empty(len(lens), device="cuda").uniform_(0.01, 0.9, generator=g))
    elif kind == "decode":
        from areal_b200.ops.lm_head import lm_head_sample, new_sampling_rng

        B = case["batch"]
        g, w, ids = _token_inputs(case, seed, B)
        model = _model(case, w, True).eval()
        ctx, table, pages = _pages(case, g)
        k, v = _caches(case, g, pages)
        caches, table, lens = list(zip(k, v)), table.cuda(), torch.tensor(ctx, dtype=torch.int32, device="cuda")
        pos = lens - 1
        slots = (torch.arange(pages - B, pages, device="cuda") * PAGE + pos % PAGE).long()
        temp, rng = torch.ones(B, device="cuda"), new_sampling_rng(seed, "cuda")

        def step():
            hidden = model.decode(ids, pos, caches, table, lens, slots, max_seq_len=case["context"])
            return (hidden, *lm_head_sample(hidden, model.output_weight(), temp, rng))

        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(stream):
            step()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                out = step()
        torch.cuda.current_stream().wait_stream(stream)
        # the inputs that the graph reads live as long as it does
        state.update(graph=graph, out=out, held=(model, ids, pos, table, lens, slots, temp, rng, k, v), pages=(k[:, pages - B:], v[:, pages - B:]))
    else:
        x, temp, u = _sample_inputs(case, seed)
        state.update(x=x, temp=temp, u=u, top_p=torch.full_like(temp, case["top_p"]) if case["top_p"] < 1 else None,
                     top_k=torch.full((case["batch"],), case["top_k"], dtype=torch.int32, device="cuda") if case["top_k"] else None)
    return state


# ---------------------------------------------------------------------------------------------------- run


def run(s):
    kind = s["kind"]
    if kind == "trunk_train":
        s["main"].zero_()
        s["x"].grad = None
        for _, p in s["named"]:
            p.grad = None
        y = s["model"](s["pos"], s["pos"], s["meta"], embeds=s["x"])
        y.backward(s["dy"])
        grads = {n: p.main_grad if p.grad is None else p.grad for n, p in s["named"]}
        return dict(hidden=y.detach(), dx=s["x"].grad, grads=grads)
    if kind == "head_train":
        from areal_b200.ops.lm_head import lm_head_logprobs
        from areal_b200.ops.rl_ops import ppo_loss_fused

        s["w"].main_grad.zero_()
        s["x"].grad = None
        logp, ent = lm_head_logprobs(s["x"], s["w"], s["labels"])
        loss, _ = ppo_loss_fused(logp, s["prox"], s["behav"], s["adv"], s["mask"], eps_clip=0.2, behav_cap=5.0, denom=s["count"])
        loss.backward()
        return dict(loss=loss.detach(), logp=logp.detach(), entropy=ent.detach(), dx=s["x"].grad, dw=s["w"].main_grad)
    if kind == "logp":
        from areal_b200.ops.lm_head import lm_head_logprobs

        with torch.no_grad():
            hidden = s["model"](s["ids"], s["pos"], s["meta"])
            logp, ent = lm_head_logprobs(hidden, s["model"].output_weight(), torch.roll(s["ids"], -1))
        return dict(hidden=hidden, logp=logp, entropy=ent)
    if kind == "prefill":
        from areal_b200.ops.rollout_ops import sample

        with torch.no_grad():
            hidden = s["model"].prefill(s["ids"], s["pos"], s["meta"], s["caches"], s["slots"])
            logits = s["model"].logits(hidden.index_select(0, s["last"]), out_dtype=torch.float32)
            tokens, logp = sample(logits, s["temp"], None, None, s["u"])
        return dict(logits=logits, tokens=tokens, logp=logp, k=s["k"], v=s["v"])
    if kind == "decode":
        s["graph"].replay()
        hidden, tokens, logp = s["out"]
        return dict(hidden=hidden, tokens=tokens, logp=logp, k=s["pages"][0], v=s["pages"][1])
    from areal_b200.ops.rollout_ops import sample

    tokens, logp = sample(s["x"], s["temp"], s["top_k"], s["top_p"], s["u"])
    return dict(tokens=tokens, logp=logp)


# ----------------------------------------------------------------------------------------------- accounting


def _layer_numbers(m):
    """Weights of one layer: all of them, and those that one token multiplies with."""
    attn = m["H"] * (m["Hq"] + 2 * m["Hkv"]) * HEAD + m["H"] * m["Hq"] * HEAD
    if m["E"]:
        return attn + m["E"] * (3 * m["Ie"] + 1) * m["H"], attn + (m["k"] * 3 * m["Ie"] + m["E"]) * m["H"]
    return attn + 3 * m["H"] * m["I"], attn + 3 * m["H"] * m["I"]


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return dict(bytes=4.0 * case["batch"] * case["vocab"], flops=4.0 * case["batch"] * case["vocab"])
    m = WIDTHS[case["model"]]
    H, V = m["H"], m["V"]
    if kind == "head_train":
        T = case["tokens"]
        return dict(bytes=V * H * (2.0 + 4.0) + 4.0 * T * H, flops=6.0 * T * H * V)
    stored, used = _layer_numbers(m)
    L = case["layers"]
    if kind == "decode":
        ctx, B = _contexts(case), case["batch"]
        cache = 4.0 * m["Hkv"] * HEAD * L * sum(ctx)
        return dict(bytes=2.0 * (L * stored + V * H) + cache, flops=2.0 * B * (L * used + V * H) + 4.0 * m["Hq"] * HEAD * L * sum(ctx))
    T, lens = case["tokens"], _lengths(case)
    pairs = sum(n * (n + 1) / 2 for n in lens)
    forward = 2.0 * T * L * used + 4.0 * m["Hq"] * HEAD * L * pairs
    if kind == "trunk_train":
        return dict(bytes=(2.0 + 4.0) * L * stored + 2.0 * 4 * T * H, flops=6.0 * T * L * used + 14.0 * m["Hq"] * HEAD * L * pairs)
    if kind == "logp":
        return dict(bytes=2.0 * (L * stored + V * H) + 2.0 * T * H, flops=forward + 2.0 * T * H * V)
    cache = 4.0 * m["Hkv"] * HEAD * L * T
    return dict(bytes=2.0 * (L * stored + V * H) + cache, flops=forward + 2.0 * len(lens) * H * V)


def tolerance(case):
    """bf16 keeps 8 bits: a rounding step is 0.4% of a value, and the passes chain several dozen of them."""
    kind = case["kind"]
    if kind == "sample":
        return dict(rel=1e-5, differ=0.01)  # fp32 sums over the vocabulary; a draw on the edge of two tokens may fall either way
    if kind == "head_train":
        return dict(rel=0.01, max=0.5)
    return dict(rel=0.03, max=0.95, differ=0.01)


# ------------------------------------------------------------------------------------- plain 64-bit statement


def _f(t):
    return t.double()


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate(x, pos):
    """``x [T, heads, 128]`` at positions ``pos``."""
    inv = THETA ** (-torch.arange(0, HEAD, 2, device=x.device, dtype=torch.float64) / HEAD)
    a = pos.double()[:, None] * inv
    c, s = a.cos()[:, None], a.sin()[:, None]
    x1, x2 = x[..., :HEAD // 2], x[..., HEAD // 2:]
    return torch.cat((x1 * c - x2 * s, x2 * c + x1 * s), -1)


def _attend(q, k, v):
    """Causal attention of one head over one sequence."""
    s = (q @ k.t()) * HEAD ** -0.5
    n = s.shape[0]
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    return s.softmax(-1) @ v


def _kept(fn, *args):
    from torch.utils.checkpoint import checkpoint

    return checkpoint(fn, *args, use_reentrant=False) if torch.is_grad_enabled() else fn(*args)


def _fp8_pair(x, w):
    """What block-scaled fp8 makes of the operands of ``x w^T`` (scales are powers of two); gradients pass straight through."""
    def quantised(t, rows):
        a = F.pad(t.detach(), (0, -t.shape[1] % 128, 0, -t.shape[0] % rows))
        b = a.view(a.shape[0] // rows, rows, a.shape[1] // 128, 128)
        scale = torch.exp2(torch.ceil(torch.log2(b.abs().amax((1, 3), keepdim=True).clamp(min=1e-12) / 448)))
        r = ((b / scale).float().to(torch.float8_e4m3fn).double() * scale).reshape(a.shape)[:t.shape[0], :t.shape[1]]
        return t + (r - t).detach()

    xq, wq = quantised(x, 1), quantised(w, 128)
    return xq.detach() @ wq.detach().t() + (x @ w.t() - (x @ w.t()).detach())


def _product(x, w, fp8):
    return _fp8_pair(x, w) if fp8 else x @ w.t()


def _experts(y, w, p, m):
    top, idx = (y @ w[p + "mlp.router"].t()).softmax(-1).topk(m["k"], -1)
    top = top / top.sum(-1, keepdim=True)
    out = torch.zeros_like(y)
    for e in range(m["E"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            g, u = (y[t] @ w[p + "mlp.gate_up"][e].t()).chunk(2, -1)
            out = out.index_add(0, t, ((F.silu(g) * u) @ w[p + "mlp.down"][e].t()) * top[t, j][:, None])
    return out


def _projected(y, w, p, m, pos):
    qkv = y @ w[p + "attn.qkv"].t()
    if not m["norm"]:
        qkv = qkv + w[p + "attn.qkv_bias"]
    q, k, v = (t.reshape(y.shape[0], -1, HEAD) for t in qkv.split([m["Hq"] * HEAD, m["Hkv"] * HEAD, m["Hkv"] * HEAD], -1))
    if m["norm"]:
        q, k = _rms(q, w[p + "attn.q_norm"]), _rms(k, w[p + "attn.k_norm"])
    return _rotate(q, pos), _rotate(k, pos), v


def _layer(x, w, p, m, pos, lens, fp8, keep=None):
    q, k, v = _projected(_rms(x, w[p + "input_norm"]), w, p, m, pos)
    if keep is not None:
        keep.append((k, v))
    rows, group = [], m["Hq"] // m["Hkv"]
    for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens)):
        rows.append(torch.stack([_kept(_attend, qs[:, h], ks[:, h // group], vs[:, h // group]) for h in range(m["Hq"])], 1))
    x = x + _product(torch.cat(rows).flatten(1), w[p + "attn.o"], fp8)
    y = _rms(x, w[p + "post_norm"])
    if m["E"]:
        return x + _experts(y, w, p, m)
    g, u = _product(y, w[p + "mlp.gate_up"], fp8).chunk(2, -1)
    return x + _product(F.silu(g) * u, w[p + "mlp.down"], fp8)


def _head_stats(x, w, labels, rows=1024):
    """Log-probabilities, entropies and log-normalisers in row chunks."""
    logp, ent = [], []
    for a, b in zip(x.split(rows), labels.split(rows)):
        z = (a @ w.t()).log_softmax(-1)
        logp.append(z.gather(1, b[:, None].long())[:, 0])
        ent.append(-(z.exp() * z).sum(-1))
        del z
    return torch.cat(logp), torch.cat(ent)


def _exact_trunk(case, seed):
    m = WIDTHS[case["model"]]
    w, x, dy = _trunk_inputs(case, seed)
    _, pos = _packed_plain(case)
    w = {n: _f(t).requires_grad_() for n, t in w.items()}
    x = _f(x).requires_grad_()
    h = x
    for i in range(case["layers"]):
        p = f"layers.{i}."
        mine = [n for n in w if n.startswith(p)]
        h = _kept(lambda h, *t, p=p, mine=mine: _layer(h, dict(zip(mine, t)), p, m, pos, _lengths(case), bool(case["fp8"])), h, *[w[n] for n in mine])
    y = _rms(h, w["norm"])
    y.backward(_f(dy))
    return dict(hidden=y.detach(), dx=x.grad, grads={n: t.grad for n, t in w.items()})


def _packed_plain(case):
    lens = _lengths(case)
    return lens, torch.cat([torch.arange(n) for n in lens]).cuda()


def _exact_head(case, seed):
    s = _head_inputs(case, seed)
    w, x, T = _f(s["w"]), _f(s["x"]), case["tokens"]
    logp, ent = _head_stats(x, w, s["labels"])
    prox, behav, adv, mask = _f(s["prox"]), _f(s["behav"]), _f(s["adv"]), s["mask"]
    lp = logp.clone().requires_grad_()
    ratio, weight = (lp - prox).exp(), (prox - behav).exp()
    per = torch.maximum(-adv * ratio, -adv * ratio.clamp(0.8, 1.2)) * weight * (mask & (weight <= 5.0))
    loss = per.sum() / mask.sum()
    loss.backward()
    dx, dw = [], torch.zeros_like(w)
    for r in range(0, T, 1024):
        a, lab = x[r:r + 1024], s["labels"][r:r + 1024].long()
        z = -(a @ w.t()).softmax(-1)
        z[torch.arange(len(lab), device="cuda"), lab] += 1
        z *= lp.grad[r:r + 1024, None]
        dx.append(z @ w)
        dw += z.t() @ a
    return dict(loss=loss.detach(), logp=logp, entropy=ent, dx=torch.cat(dx), dw=dw)


def _exact_tokens(case, seed):
    """``logp`` and ``prefill``: all layers over packed tokens."""
    m = WIDTHS[case["model"]]
    g, w, ids = _token_inputs(case, seed, case["tokens"])
    lens, pos = _packed_plain(case)
    h, kept = _f(w["embed"][ids.long()]), []
    for i in range(case["layers"]):
        p = f"layers.{i}."
        h = _layer(h, {n: _f(t) for n, t in w.items() if n.startswith(p)}, p, m, pos, lens, False, kept if case["kind"] == "prefill" else None)
    hidden, head = _rms(h, _f(w["norm"])), _f(w["embed"])
    if case["kind"] == "logp":
        logp, ent = _head_stats(hidden, head, torch.roll(ids, -1))
        return dict(hidden=hidden, logp=logp, entropy=ent)
    slots, pages = _prefill_slots(lens)
    k, v = (torch.zeros((case["layers"], pages, m["Hkv"], PAGE, HEAD), dtype=torch.float64, device="cuda") for _ in range(2))
    for i, (ki, vi) in enumerate(kept):
        k[i, slots // PAGE, :, slots % PAGE], v[i, slots // PAGE, :, slots % PAGE] = ki, vi
    last = torch.tensor([sum(lens[:i + 1]) - 1 for i in range(len(lens))], device="cuda")
    u = torch.empty(len(lens), device="cuda").uniform_(0.01, 0.9, generator=g)
    logits = hidden[last] @ head.t()
    tokens, logp = _drawn(logits, u, 0, 1.0)
    return dict(logits=logits, tokens=tokens, logp=logp, k=k, v=v)


def _exact_decode(case, seed):
    m, B = WIDTHS[case["model"]], case["batch"]
    g, w, ids = _token_inputs(case, seed, B)
    ctx, table, pages = _pages(case, g)
    kc, vc = _caches(case, g, pages)
    table, group = table.cuda().long(), m["Hq"] // m["Hkv"]
    pos = torch.tensor(ctx, device="cuda") - 1
    h, k_out, v_out = _f(w["embed"][ids.long()]), _f(kc[:, pages - B:]), _f(vc[:, pages - B:])
    every = torch.arange(B, device="cuda")
    for i in range(case["layers"]):
        p = f"layers.{i}."
        wl = {n: _f(t) for n, t in w.items() if n.startswith(p)}
        q, k, v = _projected(_rms(h, wl[p + "input_norm"]), wl, p, m, pos)
        k_out[i, every, :, pos % PAGE], v_out[i, every, :, pos % PAGE] = k, v
        rows = []
        for b, n in enumerate(ctx):
            at = table[b, :-(-n // PAGE) - 1]
            ks, vs = (torch.cat((_f(c[i, at]), o[i, b:b + 1])).transpose(1, 2).reshape(-1, m["Hkv"], HEAD)[:n].transpose(0, 1)
                      for c, o in ((kc, k_out), (vc, v_out)))
            s = (q[b].view(m["Hkv"], group, HEAD) @ ks.transpose(1, 2)) * HEAD ** -0.5
            rows.append((s.softmax(-1) @ vs).reshape(-1))
        h = h + torch.stack(rows) @ wl[p + "attn.o"].t()
        g_, u_ = (_rms(h, wl[p + "post_norm"]) @ wl[p + "mlp.gate_up"].t()).chunk(2, -1)
        h = h + (F.silu(g_) * u_) @ wl[p + "mlp.down"].t()
    hidden = _rms(h, _f(w["norm"]))
    # the drawn token depends on the kernel's own noise, but nearly always is the likeliest one
    logp, tokens = (hidden @ _f(w["embed"]).t()).log_softmax(-1).max(-1)
    return dict(hidden=hidden, tokens=tokens.int(), logp=None if (logp < -0.02).any() else logp, k=k_out, v=v_out)


def _drawn(y, u, top_k, top_p):
    """Inverse-CDF draws in vocabulary order from the kept tokens; log-probabilities before filtering."""
    z = y.log_softmax(-1)
    p = z.exp()
    keep = torch.ones_like(p, dtype=torch.bool)
    order = p.sort(-1, descending=True).values
    if top_k:
        keep &= p >= order[:, top_k - 1:top_k]
    if top_p < 1:
        count = (order.cumsum(-1) < top_p).sum(-1, keepdim=True)
        keep &= p >= order.gather(1, count)
    cdf = (p * keep).cumsum(-1)
    tokens = torch.searchsorted(cdf, (u.double() * cdf[:, -1])[:, None], right=True).clamp(max=y.shape[1] - 1)
    return tokens[:, 0].int(), z.gather(1, tokens)[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "trunk_train":
        return _exact_trunk(case, seed)
    if kind == "head_train":
        return _exact_head(case, seed)
    with torch.no_grad():
        if kind in ("logp", "prefill"):
            return _exact_tokens(case, seed)
        if kind == "decode":
            return _exact_decode(case, seed)
        x, temp, u = _sample_inputs(case, seed)
        tokens, logp = _drawn(_f(x) / _f(temp)[:, None], u, case["top_k"], case["top_p"])
        return dict(tokens=tokens, logp=logp)
