"""Workloads that stand for what this framework is used for, for timing and for comparing two builds.

Every case goes through the public entry points: ``Trainer.train_step`` (one whole optimizer step: forward,
loss, backward, gradient norm, clip, AdamW), ``gptForward`` without targets (logits), and
``eval.sample_tokens`` (generation).  The listed cases are the configurations that the repository names
(bench.py's workloads, the defaults of ``ModelConfig`` / ``TrainConfig``, the shapes of the step fixtures)
with the options that are used in earnest: fp32 (the default) and bf16 compute, both block architectures,
tied and untied heads, accumulated micro-steps, activation checkpointing, the fused route and the
reference-shaped one.  ``draw`` gives more of the same ranges, odd sequence lengths, batches and
vocabularies among them.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from alpha2_b200.autograd import Param, Tape
from alpha2_b200.backend import CudaBackend, TensorData
from alpha2_b200.data import zipf_batches
from alpha2_b200.eval import sample_tokens
from alpha2_b200.gpt import GPTParams, ModelConfig, gptForward
from alpha2_b200.rng import SeededRng
from alpha2_b200.trainer import TrainConfig, Trainer

_TRAIN = dict(kind="train", accum=1, dtype="f32", tied=True, arch="gelu", ffn=0, route="fused", ckpt=False,
              read_back=False)


def _train(name, vocab, layers, width, heads, seq, batch, **more):
    return dict(_TRAIN, name=name, vocab=vocab, layers=layers, width=width, heads=heads, block=seq, seq=seq,
                batch=batch, **more)


def listed():
    gpt2 = dict(vocab=50257, layers=12, width=768, heads=12, block=1024, dtype="bf16", tied=True, arch="gelu", ffn=0)
    return [
        # the byte-level toy that every change to a training setup is first tried on; the loss is read every
        # step, so launch latency and host time are all there is
        _train("tiny_f32_step", 256, 2, 64, 4, 64, 4, read_back=True),
        # ModelConfig() and TrainConfig() as they come: fp32, head dimension 32, untied head, batch 64
        _train("default_f32_step", 256, 6, 256, 8, 256, 64, tied=False),
        # the same model trained in bf16 with two accumulated micro-steps
        _train("default_bf16_step", 256, 6, 256, 8, 256, 32, tied=False, dtype="bf16", accum=2),
        # the small GPT of the 100-step parity runs, in both compute types
        _train("small_f32_step", 4096, 6, 384, 6, 256, 32),
        _train("small_bf16_step", 4096, 6, 384, 6, 256, 32, dtype="bf16"),
        # the headline configuration of the benchmark
        _train("gpt2_124m_bf16_step", 50257, 12, 768, 12, 1024, 16, dtype="bf16"),
        # the largest configuration: RMSNorm, SwiGLU, RoPE, untied head, four accumulated micro-steps
        _train("gpt_350m_bf16_step", 32768, 24, 1024, 16, 2048, 8, dtype="bf16", tied=False, arch="swiglu", ffn=2816,
               accum=4),
        # fine-tuning on documents of an odd length with activation checkpointing, a small batch
        dict(_train("gpt2_124m_ckpt_bf16_step", 50257, 12, 768, 12, 777, 3, dtype="bf16", ckpt=True), block=1024),
        # the op-by-op route a host takes that drives the Backend interface alone (head split and merge by
        # transposes, the flashAttention hook, unfused loss)
        _train("default_flash_f32_step", 256, 6, 256, 8, 256, 16, tied=False, route="flash"),
        # scoring text: logits of every position
        dict(gpt2, kind="logits", name="gpt2_124m_logits", seq=1024, batch=4),
        # one decision of an interactive sampler: the last position's logits of one prompt
        dict(gpt2, kind="next", name="gpt2_124m_next", seq=200, batch=1),
        # generating a passage after a prompt with the small GPT (prompt pass and token by token)
        dict(kind="sample", name="small_f32_sample", vocab=4096, layers=6, width=384, heads=6, block=256, dtype="f32",
             tied=True, arch="gelu", ffn=0, seq=48, batch=1, steps=64, topk=40),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed ranges.  fp32 models go up to the small GPT's size and bf16 ones up to the
    350M model's; head dimensions are those of the listed models (32 and 64, in fp32 16 too)."""
    most = {"f32": 3e12, "bf16": 6e13}
    while True:
        kind = rng.choices(["train", "route", "logits", "next", "sample"], [60, 10, 10, 10, 10])[0]
        dtype = "f32" if kind in ("route", "sample") else rng.choice(["f32", "bf16"])
        small = dtype == "f32"
        D = rng.choice([16, 32, 64, 64] if small else [32, 64, 64, 64])
        heads = _log(rng, max(1, 64 // D), (512 if small else 1024) // D)
        if (heads * D) % 32:
            heads += 1
        seq = _log(rng, 17, 512 if small or D != 64 else 2048)
        c = dict(vocab=_log(rng, 256, 8192 if small else 50257), layers=_log(rng, 1, 8 if small else 24),
                 width=heads * D, heads=heads, block=seq, seq=seq, dtype=dtype, tied=rng.random() < 0.6,
                 arch=rng.choice(["gelu", "gelu", "swiglu"]), ffn=0)
        if kind in ("train", "route"):
            # sampling and scoring take any batch; a step's is up to the default of 64 (bf16: 32)
            c = dict(_TRAIN, **{**c, "batch": _log(rng, 1, 64 if small else 32), "accum": rng.choice([1, 1, 1, 2, 3]),
                                "ckpt": rng.random() < 0.2, "read_back": rng.random() < 0.3})
            if kind == "route":
                c.update(route=rng.choice(["flash", "standard"]))
        elif kind == "logits":
            c.update(kind=kind, batch=_log(rng, 1, 16))
        elif kind == "next":
            c.update(kind=kind, batch=_log(rng, 1, 8))
        else:
            steps = _log(rng, 8, 96)
            c.update(kind=kind, batch=1, steps=steps, block=seq + steps, topk=rng.choice([0, 40]))
        if work(c)["flops"] <= most[dtype]:
            return c


def _config(c):
    more = dict(norm="rms", rope=True, ffnActivation="swiglu") if c["arch"] == "swiglu" else {}
    if c["ffn"]:
        more["ffnDim"] = c["ffn"]
    return ModelConfig(vocabSize=c["vocab"], blockSize=c["block"], nLayer=c["layers"], nEmbd=c["width"],
                       nHead=c["heads"], tied=c["tied"], init="plain", compute_dtype=c["dtype"], **more)


def _shapes(cfg):
    """(name, shape) of every parameter in the order of the model's own list."""
    V, T, E, F = cfg.vocabSize, cfg.blockSize, cfg.nEmbd, cfg.ffn_dim()
    norm = ["weight"] if cfg.norm == "rms" else ["weight", "bias"]
    out = [("wte", (V, E))] + ([] if cfg.rope else [("wpe", (T, E))]) + ([] if cfg.tied else [("lmHead", (V, E))])
    out += [(f"lnF.{s}", (E,)) for s in norm]
    for i in range(cfg.nLayer):
        p = f"layer.{i}"
        out += [(f"{p}.ln1.{s}", (E,)) for s in norm] + [(f"{p}.attn.wqkv", (3 * E, E)), (f"{p}.attn.wo", (E, E))]
        out += [(f"{p}.ln2.{s}", (E,)) for s in norm]
        if cfg.ffnActivation == "swiglu":
            out += [(f"{p}.mlp.fc_gate", (F, E)), (f"{p}.mlp.fc_up", (F, E)), (f"{p}.mlp.fc_proj", (E, F))]
        else:
            out += [(f"{p}.mlp.fc1", (F, E)), (f"{p}.mlp.fc2", (E, F))]
    return out


class _Part:
    """Device memory of a tensor that is a piece of one torch allocation (which it keeps alive)."""

    def __init__(self, owner, offset, nbytes):
        self.owner, self.ptr, self.nbytes = owner, owner.data_ptr() + offset, nbytes


class _Flat:
    """One fp32 torch tensor that holds a tensor of every parameter, each from a 256-byte boundary on."""

    def __init__(self, shapes):
        self.at, n = {}, 0
        for name, shape in shapes:
            self.at[name] = (n, shape)
            n += (math.prod(shape) + 63) // 64 * 64
        self.all = torch.zeros(n, dtype=torch.float32, device="cuda")

    def torch(self, name):
        n, shape = self.at[name]
        return self.all[n:n + math.prod(shape)]

    def tensor(self, name):
        n, shape = self.at[name]
        return TensorData(shape, "f32", _Part(self.all, 4 * n, 4 * math.prod(shape)))


class _View:
    """A backend tensor's device memory for torch; keeps the memory, not the tensor, alive."""

    def __init__(self, t):
        self.buf = t._buf
        kind = {"f32": "<f4", "i32": "<i4", "bf16": "<i2"}[t.dtype]
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": kind, "data": (t.ptr, False), "version": 2}


def _as_torch(t):
    out = torch.as_tensor(_View(t), device="cuda")
    return out.view(torch.bfloat16) if t.dtype == "bf16" else out


_backend = []


def prepare(case, seed):
    """The model's weights on the device (plain init, std 0.02), for training the trainer with its AdamW moments,
    and the tokens: Zipf(1.1) ids in device tensors, for sampling a prompt on the host."""
    if not _backend:
        _backend.append(CudaBackend(0))
    B, cfg = _backend[0], _config(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    shapes = _shapes(cfg)
    weights = _Flat(shapes)
    for name, shape in shapes:
        if len(shape) == 2:
            weights.torch(name).normal_(0.0, 0.02, generator=g)
        elif name.endswith(".weight"):
            weights.torch(name).fill_(1.0)
    torch.cuda.synchronize()
    P = GPTParams()
    for name, shape in shapes:
        td = weights.tensor(name)
        shadow = B.castDtype(td, "bf16") if cfg.compute_dtype == "bf16" and len(shape) == 2 else None
        P.entries[name] = Param(td, name, shadow)
    s = dict(case=case, B=B, cfg=cfg, P=P, weights=weights, seed=seed)
    if case["kind"] == "sample":
        s["prompt"] = zipf_batches(seed, 1, 1, case["seq"], case["vocab"])[0][0].reshape(-1)
        return s
    batches = zipf_batches(seed, case.get("accum", 1), case["batch"], case["seq"], case["vocab"])
    s["batches"] = [(B.upload(a, "i32"), B.upload(b, "i32")) for a, b in batches]
    if case["kind"] == "train":
        tr = Trainer(B, cfg, TrainConfig(batchSize=case["batch"], gradAccumSteps=case["accum"]), params=P,
                     attention=case["route"], activationCheckpointing=case["ckpt"])
        s["trainer"], s["m"], s["v"] = tr, _Flat(shapes), _Flat(shapes)
        for name, _ in shapes:
            tr.opt._m[name], tr.opt._v[name] = s["m"].tensor(name), s["v"].tensor(name)
    torch.cuda.synchronize()
    return s


def _logits(s, tokens, last):
    B = s["B"]
    tape = Tape()
    out = gptForward(s["cfg"], s["P"], B, tape, tokens, None, training=False, release=B.releaseGpuTensor,
                     lastOnly=last)["logits"].data
    r = _as_torch(out)
    tape.clear(B.releaseGpuTensor)
    return r


def run(state):
    """One optimizer step (the loss, the updated weights and AdamW moments), one forward (its logits), or one
    generation (the tokens, and the logits that follow them)."""
    case = state["case"]
    if case["kind"] == "train":
        r = state["trainer"].train_step(state["batches"], read_back=case["read_back"])
        loss = r["loss"] if case["read_back"] else _as_torch(r["lossTensor"])
        return {"loss": loss, "weights": state["weights"].all, "m": state["m"].all, "v": state["v"].all}
    if case["kind"] != "sample":
        return {"logits": _logits(state, state["batches"][0][0], case["kind"] == "next")}
    B = state["B"]
    tokens = sample_tokens(state["cfg"], state["P"], B, SeededRng(state["seed"]), state["prompt"], case["steps"],
                           temperature=1.0, topk=case["topk"])
    seen = B.upload(np.ascontiguousarray(tokens[-case["block"]:]).reshape(1, -1), "i32")
    return {"tokens": tokens, "logits": _logits(state, seen, True)}


def work(case):
    """Products of the matrices with every token (forward 2, forward and backward 6 operations per weight and
    token) and the causal half of the attention products; weights, and for a step the gradients' moments, read
    and written once, tokens and logits once."""
    cfg = _config(case)
    rows = case["batch"] * case["seq"]
    mats = [math.prod(s) for n, s in _shapes(cfg) if len(s) == 2 and n.startswith("layer.")]
    body, head = sum(mats), case["vocab"] * case["width"]
    total = sum(math.prod(s) for _, s in _shapes(cfg))
    size = 2 if case["dtype"] == "bf16" else 4
    att = 2.0 * case["batch"] * case["layers"] * case["seq"] ** 2 * case["width"]
    if case["kind"] == "train":
        return {"bytes": 24.0 * total + 8.0 * rows * case["accum"],
                "flops": case["accum"] * (6.0 * rows * (body + head) + 3 * att)}
    if case["kind"] == "logits":
        return {"bytes": float(size * (total + rows * case["vocab"]) + 4 * rows),
                "flops": 2.0 * rows * (body + head) + att}
    if case["kind"] == "next":
        return {"bytes": float(size * (total + case["batch"] * case["vocab"]) + 4 * rows),
                "flops": 2.0 * rows * body + 2.0 * case["batch"] * head + att}
    n = case["seq"] + case["steps"]
    return {"bytes": float(size * (total + case["vocab"]) + 4 * n),
            "flops": 2.0 * n * body + 2.0 * (case["steps"] + 1) * head
            + 2.0 * case["layers"] * float(n) ** 2 * case["width"]}


def tolerance(case):
    """fp32: the order of the sums (a weight gradient summed one by one over 16384 tokens is 2.3e-6 off its value in
    64 bits, over 65536 tokens 4.6e-6; four times that).  bf16: the rounding of activations and their gradients
    (measured against the same step in fp32: up to 7e-3 on moments and 1e-2 on logits).  Single elements of the
    moments that are sums of much larger ones differ by up to 200 times the relative error of the whole."""
    if case["dtype"] == "f32":
        return {"rel": 1.8e-5, "max": 3e-3}
    return {"rel": 0.03, "max": 0.99}


def _norm64(x, w, prefix, rms):
    if not rms:
        x = x - x.mean(-1, keepdim=True)
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w[prefix + ".weight"]
    return x if rms else x + w[prefix + ".bias"]


def _rotate64(x):
    """Rotary embedding, halves rotated, of x [B, H, T, D]."""
    T, D = x.shape[2:]
    angle = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * \
        10000.0 ** (-torch.arange(0, D, 2, dtype=torch.float64, device="cuda") / D)
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _layer64(x, w, p, heads, swiglu):
    B, T, E = x.shape
    qkv = (_norm64(x, w, p + ".ln1", swiglu) @ w[p + ".attn.wqkv"].T).view(B, T, 3, heads, E // heads)
    q, k, v = (qkv[:, :, i].transpose(1, 2) for i in range(3))
    if swiglu:
        q, k = _rotate64(q), _rotate64(k)
    s = 30.0 * torch.tanh(q @ k.transpose(-1, -2) / math.sqrt(E // heads) / 30.0)
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    x = x + (s.softmax(-1) @ v).transpose(1, 2).reshape(B, T, E) @ w[p + ".attn.wo"].T
    h = _norm64(x, w, p + ".ln2", swiglu)
    if swiglu:
        h = torch.nn.functional.silu(h @ w[p + ".mlp.fc_gate"].T) * (h @ w[p + ".mlp.fc_up"].T)
        return x + h @ w[p + ".mlp.fc_proj"].T
    h = torch.nn.functional.gelu(h @ w[p + ".mlp.fc1"].T, approximate="tanh")
    return x + h @ w[p + ".mlp.fc2"].T


def _hidden64(case, w, tokens):
    swiglu = case["arch"] == "swiglu"
    x = w["wte"][tokens]
    if not swiglu:
        x = x + w["wpe"][:tokens.shape[1]]
    for i in range(case["layers"]):
        x = torch.utils.checkpoint.checkpoint(_layer64, x, w, f"layer.{i}", case["heads"], swiglu, use_reentrant=False)
    return _norm64(x, w, "lnF", swiglu)


def exact(case, seed):
    """The same step or logits in 64 bits (from the fp32 weights, also where the layers compute in bf16).  A
    generation has no such value: one near-tie sampled otherwise changes all that follows."""
    if case["kind"] == "sample" or work(case)["flops"] > 4e13:
        return None
    g = torch.Generator(device="cuda").manual_seed(seed)
    shapes = _shapes(_config(case))
    flat = _Flat(shapes)
    for name, shape in shapes:
        if len(shape) == 2:
            flat.torch(name).normal_(0.0, 0.02, generator=g)
        elif name.endswith(".weight"):
            flat.torch(name).fill_(1.0)
    train = case["kind"] == "train"
    w = {n: flat.torch(n).double().view(s).requires_grad_(train) for n, s in shapes}
    head = w["wte"] if case["tied"] else w["lmHead"]
    batches = [tuple(torch.as_tensor(a, device="cuda").long() for a in pair)
               for pair in zipf_batches(seed, case.get("accum", 1), case["batch"], case["seq"], case["vocab"])]
    B, T, E = case["batch"], case["seq"], case["width"]
    # sequences at a time: layer inputs, one layer's intermediates and the logits within about 30 GB
    at_once = max(1, int(4e9 / (T * (E * (case["layers"] + 40) + 8 * case["heads"] * T + 4 * case["vocab"]))))
    if not train:
        with torch.no_grad():
            rows = [_hidden64(case, w, t)[:, -1:] if case["kind"] == "next" else _hidden64(case, w, t)
                    for t in batches[0][0].split(at_once)]
            return {"logits": torch.cat([r @ head.T for r in rows])}
    loss = 0.0
    for tokens, targets in batches:
        for t, y in zip(tokens.split(at_once), targets.split(at_once)):
            logits = _hidden64(case, w, t) @ head.T
            part = torch.nn.functional.cross_entropy(logits.flatten(0, 1), y.flatten(), reduction="sum")
            part = part / (B * T * case["accum"])
            part.backward()
            loss += part.item()
            del logits, part
    with torch.no_grad():
        c = TrainConfig(batchSize=B, gradAccumSteps=case["accum"])
        low, warm = c.lr / 10, min(2000, c.iters // 5)
        lr = low + (c.lr - low) / warm
        norm = math.sqrt(sum(float((p.grad ** 2).sum()) for p in w.values()))
        clip = min(1.0, c.gradClip / norm)
        out = {k: torch.zeros(flat.all.numel(), dtype=torch.float64, device="cuda") for k in ("weights", "m", "v")}
        for name, shape in shapes:
            p, d = w[name], w[name].grad * clip
            if len(shape) == 2 and name not in ("wte", "wpe"):
                p = p * (1 - lr * c.weightDecay)
            at = flat.at[name][0]
            for k, x in (("weights", p - lr * d / (d.abs() + c.eps)), ("m", (1 - c.beta1) * d),
                         ("v", (1 - c.beta2) * d * d)):
                out[k][at:at + x.numel()] = x.flatten()
    return {"loss": loss if case["read_back"] else torch.tensor([loss], dtype=torch.float64, device="cuda"), **out}
