"""The work this framework is measured on: what a user's training or evaluation program has it do on one GPU.

Most cases are whole training steps (gradients cleared, forward and backward over every micro-batch, global-norm clip,
AdamW) of the shipped model sizes with fewer layers, built and driven through the same calls as a training program.
The others are the building blocks that such programs call by themselves: decoder layers run forward only, the language
model's loss, and attention at long, short and ragged lengths.

A case is a dict of plain values; ``kind`` says which of the four it is and ``listed`` says what each stands for.
"""
import math

import torch

from hetu_galvatron_b200.core.hybrid_model import construct_hybrid_parallel_model
from hetu_galvatron_b200.core.plan import HybridPlan
from hetu_galvatron_b200.models import build_model_specs, synthetic_batch
from hetu_galvatron_b200.models.blocks import LayerBlock
from hetu_galvatron_b200.models.transformer import BatchCtx, LayerStrategy, deferred_init
from hetu_galvatron_b200.ops import autograd as A

# a learning rate of the warm-up phase; betas, decay and clip of the benchmark program
LR, OPT = 1e-5, dict(beta1=0.9, beta2=0.95, weight_decay=0.1, max_grad_norm=1.0)


def _train(name, family, size, layers, batch, chunks, seq, grads="fp32", dropout=0.0, checkpoint=False, padded=False, dec=0):
    c = {"kind": "train", "family": family, "size": size, "layers": layers, "batch": batch, "chunks": chunks, "seq": seq, "dec": dec,
         "grads": grads, "dropout": dropout, "checkpoint": checkpoint, "padded": padded}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest model anyone steps: a smoke or debugging run, where launches and host calls are the time
        _train("llama_small", "llama", "small", 2, 4, 2, 256),
        # the headline workload's layers, embedding and head: long sequences, micro-batches of two, bf16 gradient buckets
        _train("llama_7b", "llama", "llama-7b", 2, 4, 2, 4096, grads="bf16"),
        # a small decoder under activation checkpointing (every block's forward runs twice), one micro-batch
        _train("llama_0.3b_checkpoint", "llama", "llama-0.3b", 4, 4, 1, 2048, checkpoint=True),
        # decoder with head size 50, LayerNorm, biases and the training programs' default dropout of 0.1
        _train("gpt_1.5b_dropout", "gpt", "gpt-1.5b", 2, 8, 1, 1024, dropout=0.1),
        # encoder on right-padded sentences of random length, masked-token loss, head size 80
        _train("bert_huge_padded", "bert", "bert-huge-32", 2, 16, 1, 512, padded=True),
        # images of 257 tokens in the last, smaller batch of an epoch: an odd number of rows everywhere
        _train("vit_huge_ragged", "vit", "vit-huge-patch14", 2, 27, 1, 257),
        # encoder-decoder with cross attention, padded inputs, targets much shorter than inputs
        _train("t5_large_padded", "t5", "t5-large", 2, 16, 1, 512, padded=True, dec=114),
        # windowed attention with relative position bias and shifted windows, all four stages
        _train("swin_large", "swin", "swin-large-patch4-window12-384", 5, 4, 1, 9216),
        # evaluation: decoder layers forward only on one long ragged sequence, grouped key heads
        {"name": "qwen_7b_forward", "kind": "forward", "size": "qwen2.5-7b", "layers": 2, "batch": 1, "seq": 2999},
        # the loss of a model with a large vocabulary, forward and backward
        {"name": "qwen_1.5b_head", "kind": "head", "hidden": 1536, "vocab": 151936, "tokens": 2048},
        # long-context attention, forward and backward, grouped key heads
        {"name": "attention_long", "kind": "attention", "batch": 1, "sq": 16384, "sk": 16384, "hq": 32, "hk": 8, "dh": 128, "causal": True,
         "padded": False, "backward": True},
        # cross attention of one evaluation batch: short, ragged, padded keys, forward only
        {"name": "attention_short", "kind": "attention", "batch": 4, "sq": 114, "sk": 333, "hq": 16, "hk": 16, "dh": 64, "causal": False,
         "padded": True, "backward": False},
    ]


SIZES = {"llama": ["small", "llama-0.3b", "llama-7b", "qwen2.5-1.5b", "qwen2.5-3b"], "gpt": ["gpt-0.3b", "gpt-1.5b", "gpt-2.7b"],
         "bert": ["bert-base", "bert-large", "bert-huge-32"], "vit": ["vit-base", "vit-large", "vit-huge-patch14"],
         "t5": ["t5-small", "t5-base", "t5-large"], "swin": ["swin-large-patch4-window12-384", "swin-huge-patch4-window7-224"]}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 200)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "attention", "attention", "forward", "head"])
        if kind == "train":
            family = rng.choice(sorted(SIZES))
            size = rng.choice(SIZES[family])
            chunks = rng.choice([1, 1, 2])
            batch = chunks * _log(rng, 1, 24)
            seq = _log(rng, 64, 4096 if family == "llama" else 1024 if family == "gpt" else 512)
            if family in ("llama", "gpt") and rng.random() < 0.6:
                seq = max(64, seq // 64 * 64)
            c = _train(None, family, size, rng.randint(1, 3), batch, chunks, seq, rng.choice(["fp32", "bf16"]),
                       0.1 if family in ("gpt", "bert") and rng.random() < 0.5 else 0.0, rng.random() < 0.25,
                       family in ("bert", "t5") and rng.random() < 0.6, rng.randint(16, 256) if family == "t5" else 0)
            if family in ("vit", "swin"):
                c["layers"] = c["layers"] if family == "vit" else rng.randint(4, 6)
                c["seq"] = _config(c)[0].seq_length
        elif kind == "forward":
            c = {"kind": "forward", "size": rng.choice(["llama-7b", "qwen2.5-7b", "qwen2.5-1.5b", "llama-0.3b"]), "layers": rng.randint(1, 3),
                 "batch": rng.randint(1, 4), "seq": _log(rng, 32, 8192)}
        elif kind == "head":
            c = {"kind": "head", "hidden": rng.choice([1024, 1536, 2048, 4096]), "vocab": rng.choice([30592, 32000, 50304, 151936]),
                 "tokens": _log(rng, 64, 8192)}
        else:
            dh = rng.choice([40, 64, 80, 128])
            hk = rng.choice([2, 4, 8, 16])
            hq = hk * rng.choice([1, 1, 4])
            causal = rng.random() < 0.6
            sk = _log(rng, 64, 16384)
            sq = sk if causal or rng.random() < 0.5 else max(1, int(sk * rng.uniform(0.2, 1.0)))
            c = {"kind": "attention", "batch": rng.randint(1, 8), "sq": sq, "sk": sk, "hq": hq, "hk": hk, "dh": dh, "causal": causal,
                 "padded": not causal and rng.random() < 0.5, "backward": rng.random() < 0.6}
        if _cost(c) <= most:
            return c


def _config(case):
    """(model configuration, module specs) of a training or forward case."""
    family, size, kw = case.get("family", "llama"), case["size"], {}
    if size == "small":
        kw = dict(hidden_size=512, num_heads=4, num_kv_heads=2, ffn_hidden_size=1408, num_layers=case["layers"], vocab_size=4096, seq_length=case["seq"])
    else:
        kw["model_size"] = size
        if family == "swin":
            n = case["layers"]
            kw["depths"] = [1, 1, n - 3, 1]
        else:
            kw["num_layers"] = case["layers"]
        if family not in ("vit", "swin"):
            kw["seq_length"] = case["seq"]
        if family == "t5":
            kw.update(num_decoder_layers=case["layers"], decoder_seq_length=case["dec"])
    cfg, specs = build_model_specs(family, **kw)
    cfg.dropout = float(case.get("dropout", 0.0))
    return cfg, specs


def _fill(params, gen):
    """Trained-looking values: matrices of standard deviation 0.02, norm weights around 1, biases around 0."""
    for p in params:
        w = p.data
        if w.dim() >= 2:
            w.normal_(0.0, 0.02, generator=gen)
        else:
            w.add_(torch.empty_like(w).normal_(0.0, 0.02, generator=gen))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, device=dev, dtype=torch.bfloat16, generator=gen)

    kind = case["kind"]
    if kind == "train":
        cfg, specs = _config(case)
        layers = len([s for s in specs if s.layer_index is not None])
        plan = HybridPlan.from_global(layers, 1, global_bsz=case["batch"], chunks=case["chunks"], global_checkpoint=int(case["checkpoint"]))
        with deferred_init():
            model = construct_hybrid_parallel_model(cfg, plan, specs, dev, grad_dtype=torch.bfloat16 if case["grads"] == "bf16" else torch.float32)
        for b in model.engine.buckets:
            if b.numel:
                b.unshard()
                _fill(b.params, gen)
                b.commit_loaded_params()
                b.reshard()
        batch = synthetic_batch(case["family"], cfg, case["batch"], seed, dev, padded=case["padded"])
        return {"kind": kind, "model": model, "batch": batch}
    if kind == "forward":
        cfg, _ = _config(dict(case, family="llama"))
        with deferred_init():
            blocks = [LayerBlock(cfg, LayerStrategy(), i, dev) for i in range(case["layers"])]
        for blk in blocks:
            _fill(blk.parameters(), gen)
        return {"kind": kind, "blocks": blocks, "h": normal(case["seq"] * case["batch"], cfg.hidden_size), "batch": case["batch"], "seq": case["seq"]}
    if kind == "head":
        t, v = case["tokens"], case["vocab"]
        return {"kind": kind, "x": normal(t, case["hidden"]).requires_grad_(), "w": (normal(v, case["hidden"]) * 0.02).requires_grad_(),
                "labels": torch.randint(0, v, (t,), device=dev, generator=gen), "dloss": torch.full((t,), 1.0 / t, device=dev)}
    b, sq, sk, hq, hk, dh = (case[k] for k in ("batch", "sq", "sk", "hq", "hk", "dh"))
    s = {"kind": kind, "q": normal(b, sq, hq, dh), "k": normal(b, sk, hk, dh), "v": normal(b, sk, hk, dh), "causal": case["causal"], "lens": None}
    if case["padded"]:
        s["lens"] = torch.randint(max(sk // 2, 1), sk + 1, (b,), device=dev, generator=gen, dtype=torch.int32)
    if case["backward"]:
        s["do"] = normal(b, sq, hq, dh)
        for k in "qkv":
            s[k].requires_grad_()
    return s


def run(s):
    if s["kind"] == "train":
        model = s["model"]
        model.zero_grad()
        loss = model.forward_backward(s["batch"])
        norm = model.optimizer_step(LR, **OPT)
        out = {"loss": loss, "norm": norm}
        for b in model.engine.buckets:
            if b.numel:
                # the embedding bucket goes out parameter by parameter: a table of mostly untouched rows next to vectors that sum
                # over every token have no common scale to compare them on
                parts = {b.name: slice(None)}
                if b is model.engine.buckets[0]:
                    parts = {"%s.%d" % (b.name, i): slice(o, o + p.numel()) for i, (p, o) in enumerate(zip(b.params, b.offsets))}
                for name, at in parts.items():
                    out["grad." + name], out["weight." + name] = b.grad_flat[at], b.master[at]
                    out["mean." + name], out["square." + name] = b.exp_avg[at], b.exp_avg_sq[at]
        return out
    if s["kind"] == "forward":
        with torch.no_grad():
            h = s["h"]
            for blk in s["blocks"]:
                h = blk(h, BatchCtx(batch=s["batch"], seq=s["seq"]))
        return h
    if s["kind"] == "head":
        loss = A.lm_head_loss(s["x"], s["w"], s["labels"])
        return (loss.detach(),) + torch.autograd.grad(loss, (s["x"], s["w"]), s["dloss"])
    if "do" not in s:
        with torch.no_grad():
            return A.attention(s["q"], s["k"], s["v"], s["causal"], kv_lens=s["lens"])
    o, lse = A.attention(s["q"], s["k"], s["v"], s["causal"], kv_lens=s["lens"])
    return (o.detach(), lse) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])


def _layer_flops(cfg, rows, keys, batch, causal, cross_keys=0):
    """Forward multiply-adds (x 2) of one block over ``rows`` queries of each of ``batch`` sequences."""
    h, f = cfg.hidden_size, cfg.ffn_hidden_size
    kv = cfg.num_kv_heads * cfg.head_dim
    proj = h * (2 * h + 2 * kv) + h * f * (3 if cfg.act == "swiglu" else 2)
    fl = 2.0 * batch * rows * proj + 4.0 * batch * rows * keys * h * (0.5 if causal else 1.0)
    if cross_keys:
        fl += 2.0 * batch * (rows * 2 * h * h + cross_keys * 2 * h * h) + 4.0 * batch * rows * cross_keys * h
    return fl, proj + (4 * h * h if cross_keys else 0)


def work(case):
    kind = case["kind"]
    if kind == "attention":
        b, sq, sk, hq, hk, dh = (case[k] for k in ("batch", "sq", "sk", "hq", "hk", "dh"))
        fl = 4.0 * b * hq * sq * sk * dh * (0.5 if case["causal"] else 0.75 if case["padded"] else 1.0)
        q, kv = 2.0 * b * sq * hq * dh, 2.0 * b * sk * hk * dh
        by = 2 * q + 2 * kv + 4.0 * b * hq * sq
        return {"flops": fl * (3.5 if case["backward"] else 1.0), "bytes": by + (2 * q + 2 * kv if case["backward"] else 0)}
    if kind == "head":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        return {"flops": 6.0 * t * h * v, "bytes": 4.0 * (t * h + v * h) + 12.0 * t}
    cfg, specs = _config(case if kind == "train" else dict(case, family="llama"))
    b, n = case["batch"], case["layers"]
    if kind == "forward":
        fl, w = _layer_flops(cfg, case["seq"], case["seq"], b, True)
        return {"flops": n * fl, "bytes": 2.0 * n * w + 4.0 * b * case["seq"] * cfg.hidden_size}
    if case["family"] == "swin":
        from hetu_galvatron_b200.models.swin import stage_dims
        fl = par = 0.0
        for i, d in enumerate(cfg.depths):
            res, c, _ = stage_dims(cfg, i)
            w = 4 * c * c + 2 * c * c * cfg.mlp_ratio
            merge = 8 * c * c if i + 1 < len(cfg.depths) else 0
            fl += b * res * res * (d * (2.0 * w + 4.0 * min(cfg.window_size, res) ** 2 * c) + 2.0 * merge / 4)
            par += d * w + merge
    else:
        s, dec = cfg.seq_length, case["dec"]
        f1, w1 = _layer_flops(cfg, s, s, b, cfg.causal)
        fl, par = n * f1, float(n * w1)
        out_tokens = b * s
        if dec:
            f2, w2 = _layer_flops(cfg, dec, dec, b, True, cross_keys=s)
            fl, par, out_tokens = fl + n * f2, par + n * w2, b * dec
        if case["family"] == "vit":
            par += cfg.hidden_size * (cfg.hidden_size + cfg.num_labels + 3 * cfg.patch_size ** 2)
            fl += 2.0 * b * s * cfg.hidden_size * 3 * cfg.patch_size ** 2
        else:
            table = cfg.padded_vocab_size * cfg.hidden_size
            fl += 2.0 * out_tokens * table
            par += table * (1 if cfg.tie_embeddings else 2)
    # parameter read and written in bf16, fp32 master and moments read and written, gradient written once
    return {"flops": 3.0 * fl, "bytes": par * (4 + 24 + (2 if case["grads"] == "bf16" else 4))}


def tolerance(case):
    """About four times the distance of these bf16 paths from the same path in fp32, measured on the listed cases: attention
    0.0025, the head's loss gradients 0.0017, decoder layers 0.007. A training step's gradients and moments are 0.003 to 0.02 away,
    the most where 8,192 tokens meet bf16 gradient buckets, and two correct implementations up to 1.5 times that."""
    return {"rel": {"attention": 0.01, "head": 0.007, "forward": 0.025, "train": 0.03}[case["kind"]]}
