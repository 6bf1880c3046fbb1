"""The framework's main work on one GPU as a list of cases that a timing program can run.

Each case is one pass through public entry points at sizes of this repository's configurations and benchmarks:

* ``train``      one optimizer step of GPT-2 through the trainer's backend (whole-step CUDA graph, pinned tokens, loss read back)
* ``module``     loss and gradients of a BF16 `lm.LanguageModel` (Llama and GPT-2 designs) over the fused operators
* ``attention``  `fused.ops.attention`, forward and backward, on its own: long sequences, grouped heads, windows
* ``experts``    `moe.gpu.moe_ffn`, forward and backward
* ``mxfp8``      a block-scaled FP8 linear layer, forward and backward
* ``decode``     one greedy decode step of the GPT-2 serving engine: a token of every sequence, logits, the sampler
* ``prefill``    one packed step of fresh GPT-2 prompts of mixed lengths
* ``requests``   whole requests on the hybrid engine (Gugedra: windowed attention, SSD, delta rule): prompts, then some decode steps

`exact` states the same mathematics as plain torch in 64 bits, on the weights as the models hold them (BF16 where they compute in
BF16).  Weights and inputs are random: there are no checkpoints to load."""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda"
BF16 = torch.bfloat16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the headline benchmark: GPT-2 124M, 16 sequences of 1024 tokens
        dict(name="train_gpt2_124m", kind="train", layers=12, width=768, heads=12, vocab=50257, batch=16, length=1024),
        # fine-tuning a small model on short ragged sequences: launches and small GEMMs
        dict(name="train_small", kind="train", layers=4, width=256, heads=4, vocab=8192, batch=3, length=203),
        # two layers of the tinyllama-1.1b preset (RMSNorm, RoPE, grouped heads, SwiGLU), tied head
        dict(name="module_llama", kind="module", design="llama", layers=2, width=2048, heads=32, kv_heads=4, ff=5632, vocab=32000,
             batch=4, length=1024),
        # a small GPT-2 design with an odd number of rows
        dict(name="module_gpt_small", kind="module", design="gpt2", layers=2, width=512, heads=8, kv_heads=8, ff=2048, vocab=8192,
             batch=3, length=203),
        # the attention of the llama3-8b preset at 4096 tokens
        dict(name="attention_8b_4096", kind="attention", dim=128, heads=32, kv_heads=8, batch=2, length=4096, window=0),
        # one expert layer of the moe-16l-64e configuration
        dict(name="experts_64", kind="experts", experts=64, top=2, width=2048, ff=1408, rows=8192),
        # the up projection of the llama2-7b preset in block-scaled FP8
        dict(name="mxfp8_7b_up", kind="mxfp8", rows=8192, inner=4096, outer=11008),
        # continuous batching of GPT-2 XL
        dict(name="decode_xl_64", kind="decode", layers=48, width=1600, heads=25, vocab=50257, seqs=64, context=700),
        # a chat of one with GPT-2 124M: latency
        dict(name="decode_124m_1", kind="decode", layers=12, width=768, heads=12, vocab=50257, seqs=1, context=300),
        # admission of waiting requests
        dict(name="prefill_124m_32", kind="prefill", layers=12, width=768, heads=12, vocab=50257, seqs=32, longest=512),
        # requests to a hybrid design
        dict(name="requests_gugedra", kind="requests", layers=6, width=1024, seqs=8, longest=700, steps=8),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "module", "attention", "experts", "mxfp8", "decode", "prefill", "requests"])
    if kind == "train":
        layers, width, heads = rng.choice([(2, 128, 2), (4, 256, 4), (6, 384, 6), (4, 512, 4), (12, 768, 12), (6, 768, 6)])
        batch = _log(rng, 1, 16)
        return dict(kind=kind, layers=layers, width=width, heads=heads, vocab=rng.choice([512, 8192, 32000, 50257]), batch=batch,
                    length=_log(rng, 32, min(1024, 16384 // batch)))
    if kind == "module":
        design = rng.choice(["llama", "gpt2"])
        dim = rng.choice([64, 128])
        heads = rng.choice([4, 8, 12, 16])
        batch = _log(rng, 1, 8)
        return dict(kind=kind, design=design, layers=rng.choice([1, 2]), width=dim * heads, heads=heads,
                    kv_heads=rng.choice([heads, heads // 4]) if design == "llama" else heads, ff=rng.choice([2, 4]) * dim * heads,
                    vocab=rng.choice([8192, 32000]), batch=batch, length=_log(rng, 33, min(1024, 4096 // batch)))
    if kind == "attention":
        heads = rng.choice([8, 12, 16, 32])
        return dict(kind=kind, dim=rng.choice([64, 128]), heads=heads, kv_heads=rng.choice([heads, heads // 4]),
                    batch=_log(rng, 1, 4), length=_log(rng, 100, 4096), window=rng.choice([0, 0, 256, 1024]))
    if kind == "experts":
        return dict(kind=kind, experts=rng.choice([8, 16, 64]), top=rng.choice([1, 2, 4]), width=rng.choice([512, 1024, 2048]),
                    ff=rng.choice([512, 1408, 1856]), rows=_log(rng, 200, 6000))
    if kind == "mxfp8":
        return dict(kind=kind, rows=16 * _log(rng, 4, 512), inner=rng.choice([768, 2048, 4096]), outer=16 * _log(rng, 32, 688))
    if kind == "decode":
        layers, width, heads = rng.choice([(12, 768, 12), (24, 1024, 16), (36, 1280, 20)])
        return dict(kind=kind, layers=layers, width=width, heads=heads, vocab=50257, seqs=_log(rng, 1, 100),
                    context=_log(rng, 20, 700))
    if kind == "prefill":
        layers, width, heads = rng.choice([(12, 768, 12), (24, 1024, 16)])
        seqs = _log(rng, 1, 48)
        return dict(kind=kind, layers=layers, width=width, heads=heads, vocab=50257, seqs=seqs, longest=_log(rng, 24, min(1000, 16384 // seqs)))
    return dict(kind="requests", layers=rng.choice([3, 6]), width=1024, seqs=_log(rng, 1, 12), longest=_log(rng, 20, 600),
                steps=rng.randint(2, 8))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000 + seed)


def _randn(g, *shape, std=1.0):
    return torch.randn(*shape, device=DEV, generator=g) * std


def _lengths(longest, seqs, seed):
    """Mixed lengths between a quarter of the longest and the longest, the longest among them."""
    r = np.random.RandomState(seed + 7)
    out = r.randint(max(1, longest // 4), longest + 1, seqs)
    out[0] = longest
    return [int(n) for n in out]


def _tokens(vocab, n, seed):
    return np.random.RandomState(seed + 11).randint(0, vocab, n).astype(np.int32)


def _gpt2_config(c):
    from nexus_b200.lm.config import LmConfig
    return LmConfig(name="gpt2", vocab_size=c["vocab"], n_layer=c["layers"], d_model=c["width"], n_head=c["heads"], d_ff=4 * c["width"],
                    max_position=1024, norm="layernorm", mlp="gelu", pos="learned", tie_embeddings=True, bias=True, init="gpt2")


def _module_config(c, seed):
    from nexus_b200.lm.config import LmConfig
    common = dict(vocab_size=c["vocab"], n_layer=c["layers"], d_model=c["width"], n_head=c["heads"], n_kv_head=c["kv_heads"],
                  d_ff=c["ff"], max_position=2048, seed=seed, tie_embeddings=True)
    if c["design"] == "llama":
        return LmConfig(name="llama", norm="rmsnorm", mlp="swiglu", pos="rope", init="llama", **common)
    return LmConfig(name="gpt2", norm="layernorm", mlp="gelu", pos="learned", bias=True, init="gpt2", **common)


def _module(c, seed):
    from nexus_b200.lm.model import LanguageModel
    m = LanguageModel(_module_config(c, seed)).to(DEV).to(BF16)
    g = _gen(seed)
    with torch.no_grad():         # norms and biases away from their initial ones and zeros
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(_randn(g, *p.shape, std=0.02).to(BF16))
    m.train()
    return m


def _gpt2_weights(c, seed):
    """GPT-2 weights on the device, already rounded to BF16, all biases and norms live."""
    from nexus_b200.infer import Gpt2Weights
    g = _gen(seed)
    d, L = c["width"], c["layers"]

    def n(*shape, std=0.02):
        return _randn(g, *shape, std=std).to(BF16).float()
    w = Gpt2Weights(L, c["heads"], d, c["vocab"], 1024, n(c["vocab"], d), n(1024, d), 1 + n(d), n(d))
    ps = 0.02 / math.sqrt(2 * L)
    for _ in range(L):
        w.h.append({"ln1_w": 1 + n(d), "ln1_b": n(d), "attn_w": n(3 * d, d, std=0.05), "attn_b": n(3 * d), "proj_w": n(d, d, std=ps),
                    "proj_b": n(d), "ln2_w": 1 + n(d), "ln2_b": n(d), "fc_w": n(4 * d, d), "fc_b": n(4 * d),
                    "fc2_w": n(d, 4 * d, std=ps), "fc2_b": n(d)})
    return w


def _gugedra(c, seed):
    from nexus_b200.bench.hybrid import hybrid_config
    from nexus_b200.lm.hybrid import HybridWeights, gugedra_tensors
    cfg = hybrid_config(c["width"], c["layers"], 64)
    g, out = _gen(seed), {}
    for name, shape in gugedra_tensors(cfg).items():
        leaf = name.rsplit(".", 1)[-1]
        if leaf.startswith("norm") or leaf == "D":
            v = 1 + _randn(g, *shape, std=0.1)
        elif leaf == "A_log":
            v = torch.linspace(-1.0, 1.5, shape[0], device=DEV)
        elif leaf == "dt_bias":
            v = torch.linspace(-4.0, -1.0, shape[0], device=DEV)
        elif leaf == "b" and len(shape) == 1:
            v = _randn(g, *shape, std=0.1)
        elif leaf == "embed":
            v = _randn(g, *shape)
        else:
            v = _randn(g, *shape, std=1.0 / math.sqrt(shape[-1]))
        out[name] = v.to(BF16)
    return HybridWeights(cfg, out)


def _capacity(c):
    per = 1.25 * c["rows"] * c["top"] / c["experts"]
    return (int(math.ceil(per)) + 7) // 8 * 8


def _experts_inputs(c, seed):
    g = _gen(seed)
    N, E, d, F = c["rows"], c["experts"], c["width"], c["ff"]
    return dict(x=_randn(g, N, d).to(BF16), router=_randn(g, E, d, std=1 / math.sqrt(d)).to(BF16),
                up=_randn(g, E, 2 * F, d, std=1 / math.sqrt(d)).to(BF16), down=_randn(g, E, d, F, std=1 / math.sqrt(F)).to(BF16),
                dy=_randn(g, N, d).to(BF16))


def _attention_inputs(c, seed):
    g = _gen(seed)
    B, T, H, G, D = c["batch"], c["length"], c["heads"], c["kv_heads"], c["dim"]
    return [_randn(g, B, T, n, D).to(BF16) for n in (H, G, G, H)]


def _mxfp8_inputs(c, seed):
    g = _gen(seed)
    return (_randn(g, c["rows"], c["inner"]).to(BF16), _randn(g, c["outer"], c["inner"], std=1 / math.sqrt(c["inner"])).to(BF16),
            _randn(g, c["rows"], c["outer"]).to(BF16))


def _leaf(t):
    return t.detach().clone().requires_grad_(True)


DECODE_STEPS = 256     # decode states go back to their first context after this many steps


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c)
    if kind == "train":
        from nexus_b200.train.gpt_backend import GptLmBackend
        from nexus_b200.train.lm_trainer import AdamW
        s["backend"] = GptLmBackend(_gpt2_config(c), c["batch"], c["length"], device="cuda", seed=seed)
        s["backend"].compile(True)
        s["opt"] = AdamW(lr=6e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)
        s["tokens"] = _tokens(c["vocab"], (4, c["batch"], c["length"]), seed)
        s["at"] = 0
    elif kind == "module":
        s["model"] = _module(c, seed)
        s["tokens"] = torch.from_numpy(_tokens(c["vocab"], (c["batch"], c["length"]), seed)).to(DEV)
    elif kind == "attention":
        q, k, v, do = _attention_inputs(c, seed)
        s.update(q=_leaf(q), k=_leaf(k), v=_leaf(v), do=do)
    elif kind == "experts":
        s.update({n: (t if n == "dy" else _leaf(t)) for n, t in _experts_inputs(c, seed).items()})
        s["capacity"] = _capacity(c)
    elif kind == "mxfp8":
        x, w, dy = _mxfp8_inputs(c, seed)
        s.update(x=_leaf(x), w=_leaf(w), dy=dy)
    elif kind == "decode":
        from nexus_b200.infer import Chunk, Engine, EngineConfig, SamplingParams
        lens = _lengths(c["context"], c["seqs"], seed)
        eng = Engine(_gpt2_weights(c, seed), EngineConfig(max_seqs=c["seqs"], max_tokens=8192,
                                                          kv_tokens=sum((n + DECODE_STEPS + 31) // 16 * 16 for n in lens)))
        prompts = [_tokens(c["vocab"], n, seed + 100 * i).tolist() for i, n in enumerate(lens)]
        ids = [eng.add_sequence() for _ in lens]
        step, room = [], 8192
        for q, p in zip(ids, prompts):
            if len(p) > room:
                eng.forward(step)
                step, room = [], 8192
            step.append(Chunk(q, p, 0))
            room -= len(p)
        eng.forward(step)
        s.update(engine=eng, ids=ids, lens=lens, at=0, tokens=_tokens(c["vocab"], (DECODE_STEPS, c["seqs"]), seed + 3).tolist(),
                 params=[SamplingParams(temperature=0.0)] * c["seqs"], rows=torch.arange(c["seqs"], device=DEV))
    elif kind == "prefill":
        from nexus_b200.infer import Engine, EngineConfig
        lens = _lengths(c["longest"], c["seqs"], seed)
        s["engine"] = Engine(_gpt2_weights(c, seed), EngineConfig(max_seqs=c["seqs"], max_tokens=16384,
                                                                  kv_tokens=sum((n + 31) // 16 * 16 for n in lens)))
        s["prompts"] = [_tokens(c["vocab"], n, seed + 100 * i).tolist() for i, n in enumerate(lens)]
    else:
        from nexus_b200.infer import EngineConfig, create_engine
        lens = _lengths(c["longest"], c["seqs"], seed)
        s["engine"] = create_engine(_gugedra(c, seed), EngineConfig(
            max_seqs=c["seqs"], max_tokens=16384, context=1024, kv_tokens=sum((n + c["steps"] + 31) // 16 * 16 for n in lens)))
        s["prompts"] = [_tokens(32000, n, seed + 100 * i).tolist() for i, n in enumerate(lens)]
        s["after"] = _tokens(32000, (c["steps"], c["seqs"]), seed + 3).tolist()
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "train":
        be = s["backend"]
        be.micro_step(s["tokens"][s["at"] % 4], 1.0, 0, 1)
        be.optimizer_step(s["opt"], 6e-4, 1.0)
        res = be.finish_step()
        s["at"] += 1
        m = be.model
        return dict(loss=res.loss, grad_norm=res.grad_norm, weights=m.params, m=m.m, v=m.v)
    if kind == "module":
        m = s["model"]
        for p in m.parameters():
            p.grad = None
        loss = m.loss(s["tokens"])
        loss.backward()
        return dict(loss=loss.detach(), **{n: p.grad for n, p in m.named_parameters()})
    if kind == "attention":
        from nexus_b200.fused import ops
        o = ops.attention(s["q"], s["k"], s["v"], causal=True, window=c["window"])
        dq, dk, dv = torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])
        return dict(o=o.detach(), dq=dq, dk=dk, dv=dv)
    if kind == "experts":
        from nexus_b200.moe import gpu
        y, counts, dropped = gpu.moe_ffn(s["x"], s["router"], s["up"], s["down"], c["top"], s["capacity"])
        g = torch.autograd.grad(y, (s["x"], s["router"], s["up"], s["down"]), s["dy"])
        return dict(y=y.detach(), dx=g[0], drouter=g[1], dup=g[2], ddown=g[3])
    if kind == "mxfp8":
        from nexus_b200.fused import ops
        with ops.linear_precision("mxfp8"):
            y = ops.fused_linear(s["x"], s["w"])
            dx, dw = torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])
        return dict(y=y.detach(), dx=dx, dw=dw)
    from nexus_b200.infer import Chunk
    eng = s["engine"]
    if kind == "decode":
        if s["at"] == DECODE_STEPS:
            for q, n in zip(s["ids"], s["lens"]):
                eng.truncate(q, n)
            s["at"] = 0
        logits = eng.forward([Chunk(q, [t], 1, True) for q, t in zip(s["ids"], s["tokens"][s["at"]])])
        picked = eng.sample(s["params"], s["ids"], s["at"])
        s["at"] += 1
        return dict(logits=logits[:, : c["vocab"]], picked=logits[s["rows"], torch.tensor(picked).to(DEV, non_blocking=True)])
    ids = [eng.add_sequence() for _ in s["prompts"]]
    out = [eng.forward([Chunk(q, p, 1) for q, p in zip(ids, s["prompts"])])]
    if kind == "requests":
        for row in s["after"]:
            out.append(eng.forward([Chunk(q, [t], 1, True) for q, t in zip(ids, row)]).clone())
    for q in ids:
        eng.free_sequence(q)
    return [x[:, : eng.vocab()] for x in out]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _gpt2_matrix(c):
    return c["layers"] * 12 * c["width"] ** 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        d, L, V = c["width"], c["layers"], c["vocab"]
        n, rows = _gpt2_matrix(c) + (V + 1024) * d, c["batch"] * c["length"]
        flops = 6 * rows * (_gpt2_matrix(c) + V * d) + 3.5 * 2 * L * d * c["batch"] * c["length"] ** 2
        # masters, moments in and out; weights and gradients of the two passes; activations of every layer out and in
        return dict(bytes=n * (24 + 2 + 8 + 2) + rows * L * d * 2 * 2 * 12, flops=flops)
    if kind == "module":
        d, G, D = c["width"], c["kv_heads"], c["width"] // c["heads"]
        mat = c["layers"] * (d * (d + 2 * G * D) + d * d + (3 if c["design"] == "llama" else 2) * d * c["ff"])
        rows = c["batch"] * c["length"]
        return dict(bytes=(mat + c["vocab"] * d) * 6 + rows * c["layers"] * d * 2 * 2 * 12,
                    flops=6 * rows * (mat + c["vocab"] * d) + 3.5 * 2 * c["layers"] * d * rows * c["length"])
    if kind == "attention":
        T, W = c["length"], c["window"] or c["length"]
        keys = T * (T + 1) / 2 if W >= T else W * (W + 1) / 2 + (T - W) * W
        q, kv = (c["batch"] * T * n * c["dim"] * 2 for n in (c["heads"], c["kv_heads"]))
        return dict(bytes=4 * q + 4 * kv, flops=14 * c["batch"] * c["heads"] * keys * c["dim"])
    if kind == "experts":
        w = c["experts"] * 3 * c["width"] * c["ff"]
        return dict(bytes=4 * w + 4 * 2 * c["rows"] * c["width"], flops=18 * c["rows"] * c["top"] * c["width"] * c["ff"])
    if kind == "mxfp8":
        m, k, n = c["rows"], c["inner"], c["outer"]
        return dict(bytes=2 * (2 * m * k + 2 * m * n + 2 * n * k), flops=6 * m * n * k)
    if kind in ("decode", "prefill"):
        d, V = c["width"], c["vocab"]
        most = c["context"] if kind == "decode" else c["longest"]
        past = c["seqs"] * most * 5 / 8               # lengths are spread between a quarter and all of the longest
        weights = _gpt2_matrix(c) + V * d
        if kind == "decode":
            return dict(bytes=2 * weights + past * c["layers"] * 4 * d + c["seqs"] * V * 4,
                        flops=2 * c["seqs"] * weights + 4 * past * c["layers"] * d)
        return dict(bytes=2 * weights + past * c["layers"] * 4 * d + c["seqs"] * V * 4,
                    flops=2 * past * _gpt2_matrix(c) + 2 * c["seqs"] * V * d + 2 * past * most * 0.7 * c["layers"] * d)
    d, L, V = c["width"], c["layers"], 32000
    per = 2 * L / 3 * (d * (1.5 * d + 2 * d + 256 + d / 64) + 2 * d * d) + L / 3 * (d * (2 * d + d) + d * d) + L * (8.25 * d * d + 256 * d)
    rows = c["seqs"] * c["longest"] * 5 / 8
    return dict(bytes=2 * (c["steps"] + 1) * (per + V * d) + rows * L * d * 2, flops=2 * per * (rows + c["seqs"] * c["steps"])
                + 2 * V * d * c["seqs"] * (c["steps"] + 1))


def tolerance(case):
    """About four times the distance from the 64-bit result that one correct BF16 path was measured at (train 0.006, module 0.013,
    attention 0.0025, experts 0.0044, decode 0.02 with 48 layers and 0.004 with 12, prefill 0.0055, requests 0.012).  Block-scaled
    FP8 quantises bit for bit; beside that only the BF16 rounding of the results (0.0025) is free."""
    return dict(train={"rel": 0.025}, module={"rel": 0.05}, attention={"rel": 0.01}, experts={"rel": 0.018}, mxfp8={"rel": 0.01},
                decode={"rel": 0.08 if case.get("layers", 0) > 24 else 0.03}, prefill={"rel": 0.022}, requests={"rel": 0.05})[case["kind"]]


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _ln(x, w, b, eps=1e-5):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, eps)


def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v, scale, window=0, softcap=0.0):
    """q [B, T, H, D], k / v [B, T, G, D] -> [B, T, H, D]; one sequence and KV head at a time to bound the memory."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    i = torch.arange(T, device=q.device)
    hide = i[None] > i[:, None]
    if window:
        hide = hide | (i[None] <= i[:, None] - window)
    out = []
    for b in range(B):
        row = []
        for g in range(G):
            s = torch.einsum("thd,sd->hts", q[b, :, g * (H // G): (g + 1) * (H // G)], k[b, :, g]) * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            row.append(torch.einsum("hts,sd->thd", s.masked_fill(hide, -math.inf).softmax(-1), v[b, :, g]))
        out.append(torch.cat(row, 1))
    return torch.stack(out)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _gpt2_hidden(tokens, wte, wpe, layers, heads):
    """Residual stream after the last layer; tokens [B, T]; layers: dicts in the engine's names."""
    B, T = tokens.shape
    d = wte.shape[1]
    x = wte[tokens] + wpe[:T]
    for w in layers:
        qkv = (_ln(x, w["ln1_w"], w["ln1_b"]) @ w["attn_w"].t() + w["attn_b"]).view(B, T, 3, heads, d // heads)
        o = _attend(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], (d // heads) ** -0.5)
        x = x + o.reshape(B, T, d) @ w["proj_w"].t() + w["proj_b"]
        x = x + _gelu(_ln(x, w["ln2_w"], w["ln2_b"]) @ w["fc_w"].t() + w["fc_b"]) @ w["fc2_w"].t() + w["fc2_b"]
    return x


def _shifted_loss(logits, tokens):
    return torch.nn.functional.cross_entropy(logits[:, :-1].reshape(-1, logits.shape[-1]), tokens[:, 1:].reshape(-1), reduction="sum")


def _exact_train(c, seed):
    from nexus_b200.models.gpt import DECAY, PARAM_ORDER, GptModel
    m = GptModel(_gpt2_config(c), device="cuda", seed=seed)
    tokens = torch.from_numpy(_tokens(c["vocab"], (4, c["batch"], c["length"]), seed)[0]).long().to(DEV)
    low = {"wte", "wpe", "qkv_w", "attproj_w", "fc_w", "fcproj_w", "qkv_b", "attproj_b", "fc_b", "fcproj_b"}   # read in BF16
    p = {n: (m.w if n in low else m.p)[n].double().requires_grad_(True) for n in PARAM_ORDER}
    names = dict(ln1_w="ln1_w", ln1_b="ln1_b", attn_w="qkv_w", attn_b="qkv_b", proj_w="attproj_w", proj_b="attproj_b", ln2_w="ln2_w",
                 ln2_b="ln2_b", fc_w="fc_w", fc_b="fc_b", fc2_w="fcproj_w", fc2_b="fcproj_b")
    total, count = 0.0, c["batch"] * (c["length"] - 1)
    for b in range(c["batch"]):
        t = tokens[b: b + 1]
        x = _gpt2_hidden(t, p["wte"][: m.V], p["wpe"], [{k: p[n][l] for k, n in names.items()} for l in range(m.L)], m.H)
        loss = _shifted_loss(_ln(x, p["lnf_w"], p["lnf_b"]) @ p["wte"][: m.V].t(), t) / count
        loss.backward()
        total += float(loss)
    flat = lambda: torch.zeros(m.num_params, dtype=torch.float64, device=DEV)  # noqa: E731
    w, g, decay = m.params.double(), flat(), flat()
    for n in PARAM_ORDER:
        o, k = m.offsets[n], math.prod(m.shapes[n])
        g[o: o + k] = p[n].grad.reshape(-1)
        decay[o: o + k] = 0.1 if n in DECAY else 0.0
    norm = float(g.norm())
    g *= min(1.0, 1.0 / (norm + 1e-6))
    mm, vv = 0.1 * g, 0.05 * g * g
    w = w * (1 - 6e-4 * decay) - 6e-4 * (mm / 0.1) / ((vv / 0.05).sqrt() + 1e-8)
    return dict(loss=total, grad_norm=norm, weights=w, m=mm, v=vv)


def _exact_module(c, seed):
    m = _module(c, seed)
    cfg = m.config
    tokens = torch.from_numpy(_tokens(c["vocab"], (c["batch"], c["length"]), seed)).long().to(DEV)
    p = {n: t.detach().double().requires_grad_(True) for n, t in m.named_parameters()}
    B, T = tokens.shape
    H, G, D = cfg.n_head, cfg.kv_heads(), cfg.hdim()
    llama = c["design"] == "llama"

    def lin(x, n):
        y = x @ p[n + ".weight"].t()
        return y + p[n + ".bias"] if n + ".bias" in p else y

    def norm(x, n):
        return _rms(x, p[n + ".weight"], cfg.norm_eps) if llama else _ln(x, p[n + ".weight"], p[n + ".bias"], cfg.norm_eps)
    x = p["wte"][tokens]
    if not llama:
        x = x + p["wpe"][:T]
    ang = torch.arange(T, dtype=torch.float64, device=DEV)[:, None] * cfg.rope_theta ** (
        -torch.arange(0, D, 2, dtype=torch.float64, device=DEV) / D)
    cos, sin = (f(ang)[:, None] for f in (torch.cos, torch.sin))

    def turn(t):
        if not llama:
            return t
        a, b = t[..., : D // 2], t[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    for l in range(cfg.n_layer):
        q, k, v = lin(norm(x, f"h.{l}.norm1"), f"h.{l}.attn.qkv").split([H * D, G * D, G * D], -1)
        o = _attend(turn(q.view(B, T, H, D)), turn(k.view(B, T, G, D)), v.view(B, T, G, D), D ** -0.5)
        x = x + lin(o.reshape(B, T, H * D), f"h.{l}.attn.o")
        u = lin(norm(x, f"h.{l}.norm2"), f"h.{l}.mlp.up")
        u = torch.nn.functional.silu(u[..., : c["ff"]]) * u[..., c["ff"]:] if llama else _gelu(u)
        x = x + lin(u, f"h.{l}.mlp.down")
    loss = _shifted_loss(norm(x, "norm_f") @ p["wte"].t(), tokens) / (B * (T - 1))
    loss.backward()
    return dict(loss=loss.detach(), **{n: t.grad for n, t in p.items()})


def _exact_attention(c, seed):
    q, k, v, do = _attention_inputs(c, seed)
    B, G, H = c["batch"], c["kv_heads"], c["heads"]
    out = dict(o=torch.empty_like(q, dtype=torch.float64))
    out.update(dq=torch.empty_like(out["o"]), dk=torch.empty_like(k, dtype=torch.float64), dv=torch.empty_like(v, dtype=torch.float64))
    r = H // G
    for b in range(B):
        for g in range(G):
            h = slice(g * r, (g + 1) * r)
            x = [t.double().requires_grad_(True) for t in (q[b: b + 1, :, h], k[b: b + 1, :, g: g + 1], v[b: b + 1, :, g: g + 1])]
            o = _attend(*x, c["dim"] ** -0.5, c["window"])
            dq, dk, dv = torch.autograd.grad(o, x, do[b: b + 1, :, h].double())
            out["o"][b, :, h], out["dq"][b, :, h] = o[0].detach(), dq[0]
            out["dk"][b, :, g], out["dv"][b, :, g] = dk[0, :, 0], dv[0, :, 0]
    return out


def _exact_experts(c, seed):
    t = _experts_inputs(c, seed)
    x, router, up, down = (t[n].double().requires_grad_(True) for n in ("x", "router", "up", "down"))
    N, E, k, F, cap = c["rows"], c["experts"], c["top"], c["ff"], _capacity(c)
    val, idx = torch.sort(x @ router.t(), dim=-1, descending=True, stable=True)
    gate, idx = val[:, :k].softmax(-1), idx[:, :k]
    # places go by choice, then by token; what finds its expert full is dropped
    flat = idx.t().reshape(-1)
    order = torch.argsort(flat, stable=True)
    first = torch.searchsorted(flat[order].contiguous(), torch.arange(E, device=DEV))
    place = torch.empty_like(flat)
    place[order] = torch.arange(N * k, device=DEV) - first[flat[order]]
    keep = (place < cap).view(k, N).t()
    y = torch.zeros_like(x)
    for e in range(E):
        tok, ch = ((idx == e) & keep).nonzero(as_tuple=True)
        if tok.numel():
            h = x[tok] @ up[e].t()
            y = y.index_add(0, tok, ((torch.nn.functional.silu(h[:, :F]) * h[:, F:]) @ down[e].t()) * gate[tok, ch][:, None])
    g = torch.autograd.grad(y, (x, router, up, down), t["dy"].double())
    return dict(y=y.detach(), dx=g[0], drouter=g[1], dup=g[2], ddown=g[3])


def _exact_mxfp8(c, seed):
    x, w, dy = (t.double() for t in _mxfp8_inputs(c, seed))
    return dict(y=x @ w.t(), dx=dy @ w, dw=dy.t() @ x)


def _exact_gpt2(c, seed, lens, extra):
    """Logits of the last token of every sequence: its prompt and, where given, one token more."""
    w = _gpt2_weights(c, seed)
    d64 = lambda t: t.to(DEV).double()  # noqa: E731
    layers = [{k: d64(t) for k, t in h.items()} for h in w.h]
    wte, wpe, lw, lb = d64(w.wte), d64(w.wpe), d64(w.ln_f_w), d64(w.ln_f_b)
    out = []
    for i, n in enumerate(lens):
        t = _tokens(c["vocab"], n, seed + 100 * i).tolist() + ([extra[i]] if extra else [])
        x = _gpt2_hidden(torch.tensor(t, device=DEV)[None], wte, wpe, layers, c["heads"])
        out.append(_ln(x[0, -1], lw, lb) @ wte.t())
    return torch.stack(out)


def _exact_requests(c, seed):
    """All sequences side by side, padded at the end (nothing looks ahead), the recurrences token by token."""
    W = _gugedra(c, seed)
    cfg = W.config
    w = {n: t.double() for n, t in W.tensors.items()}
    lens = _lengths(c["longest"], c["seqs"], seed)
    after = _tokens(32000, (c["steps"], c["seqs"]), seed + 3)
    B, T = len(lens), max(lens) + c["steps"]
    tok = torch.zeros(B, T, dtype=torch.long)
    for i, n in enumerate(lens):
        tok[i, : n + c["steps"]] = torch.from_numpy(np.concatenate([_tokens(32000, n, seed + 100 * i), after[:, i]]).astype(np.int64))
    tok = tok.to(DEV)
    silu, soft = torch.nn.functional.silu, torch.nn.functional.softplus
    eps, side = cfg.norm_eps, cfg.token_side

    def conv(x, k, b=None):
        y = torch.nn.functional.conv1d(torch.nn.functional.pad(x.transpose(1, 2), (k.shape[1] - 1, 0)), k[:, None], b, groups=k.shape[0])
        return silu(y.transpose(1, 2))

    def rotate(x, dims, base):
        half = dims // 2
        ang = torch.arange(T, dtype=torch.float64, device=DEV)[:, None] * float(base) ** (
            -2.0 * torch.arange(half, dtype=torch.float64, device=DEV) / dims)
        cos, sin = ang.cos()[:, None], ang.sin()[:, None]
        a, b = x[..., :half], x[..., half: dims]
        return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., dims:]], -1)

    def parallel(h, p, m):
        a, r = m.left, m.right
        q = rotate((h @ p["left.q"].t()).view(B, T, a.heads, a.dim), a.rope_dims, a.rope_base)
        k = rotate((h @ p["left.k"].t()).view(B, T, a.kv_heads, a.dim), a.rope_dims, a.rope_base)
        v = (h @ p["left.v"].t()).view(B, T, a.kv_heads, a.vdim)
        left = _attend(q, k, v, a.scale, a.window, a.softcap).reshape(B, T, -1) @ p["left.o"].t()
        z, xbc, dt = (h @ p["right.in"].t()).split([r.inner, r.channels, r.heads], -1)
        x, bb, cc = conv(xbc, p["right.conv"], p["right.conv.b"]).split([r.inner, r.groups * r.state, r.groups * r.state], -1)
        x = x.reshape(B, T, r.heads, r.vdim)
        bb, cc = (t.reshape(B, T, r.groups, r.state).repeat_interleave(r.heads // r.groups, 2) for t in (bb, cc))
        dt = soft(dt + p["right.dt_bias"])
        keep = torch.exp(-torch.exp(p["right.A_log"]) * dt)
        S, y = x.new_zeros(B, r.heads, r.state, r.vdim), torch.empty_like(x)
        for t in range(T):
            S = keep[:, t, :, None, None] * S + (dt[:, t, :, None] * bb[:, t])[..., None] * x[:, t, :, None]
            y[:, t] = (cc[:, t, :, None] @ S)[:, :, 0]
        u = (y + p["right.D"][:, None] * x).reshape(B, T, r.inner) * silu(z)
        u = u.view(B, T, r.norm_groups, -1)
        u = (u * torch.rsqrt(u.square().mean(-1, keepdim=True) + eps)).reshape(B, T, r.inner) * p["right.norm"]
        return m.left_scale * left + m.right_scale * (u @ p["right.o"].t())

    def delta(h, p, m):
        q, k, v = (conv(h @ p[n].t(), p[n + ".conv"]) for n in ("q", "k", "v"))
        unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + m.unit_eps)  # noqa: E731
        rep = m.heads // m.kv_heads
        q = (unit(q.view(B, T, m.kv_heads, m.dim)) * m.dim ** -0.5).repeat_interleave(rep, 2)
        k, v = unit(k.view(B, T, m.kv_heads, m.dim)).repeat_interleave(rep, 2), v.view(B, T, m.heads, m.vdim)
        beta = torch.sigmoid(h @ p["b"].t())
        keep = torch.exp(-torch.exp(p["A_log"]) * soft(h @ p["a"].t() + p["dt_bias"]))
        S, o = h.new_zeros(B, m.heads, m.dim, m.vdim), torch.empty_like(v)
        for t in range(T):
            S = keep[:, t, :, None, None] * S
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
            S = S + k[:, t, :, :, None] * u[:, :, None]
            o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        o = _rms(o, p["norm"], eps) * silu((h @ p["g"].t()).view(B, T, m.heads, m.vdim))
        return o.reshape(B, T, -1) @ p["o"].t()
    x = w["embed"][tok]
    for i, layer in enumerate(cfg.layers):
        p = {n[len(f"l{i}."):]: t for n, t in w.items() if n.startswith(f"l{i}.")}
        mix = {n[4:]: t for n, t in p.items() if n.startswith("mix.")}
        mixer = parallel if hasattr(layer.mixer, "left") else delta
        x = x + _rms(mixer(_rms(x, p["norm1"], eps), mix, layer.mixer), p["norm1b"], eps)
        h = _rms(x, p["norm2"], eps)
        x = x + _rms((silu(h @ p["mlp.gate"].t()) * (h @ p["mlp.up"].t())) @ p["mlp.down"].t(), p["norm2b"], eps)
        e = w["side.embed"][tok][..., i * side: (i + 1) * side]
        x = x + _rms((_gelu(x @ p["side.gate"].t()) * e) @ p["side.proj"].t(), p["side.norm"], eps)
    at = torch.tensor(lens, device=DEV)
    cap = cfg.logit_softcap
    return [cap * torch.tanh(_rms(x[torch.arange(B, device=DEV), at - 1 + j], w["final.norm"], eps) @ w["head"].t() / cap)
            for j in range(c["steps"] + 1)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _exact_train(c, seed)
    if kind == "module":
        return _exact_module(c, seed)
    if kind == "attention":
        return _exact_attention(c, seed)
    if kind == "experts":
        return _exact_experts(c, seed)
    if kind == "mxfp8":
        return _exact_mxfp8(c, seed)
    with torch.no_grad():
        if kind == "decode":
            logits = _exact_gpt2(c, seed, _lengths(c["context"], c["seqs"], seed), _tokens(c["vocab"], (DECODE_STEPS, c["seqs"]), seed + 3)[0].tolist())
            return dict(logits=logits, picked=logits.amax(1))
        if kind == "prefill":
            return [_exact_gpt2(c, seed, _lengths(c["longest"], c["seqs"], seed), None)]
        return _exact_requests(c, seed)
