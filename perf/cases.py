"""The work whose speed this repository is measured by.

A case is one call (or one pass of calls) that a user's program makes through the package's public entry
points, at a size from the range that such programs meet.  `listed()` names the cases, `draw(rng)` gives
further ones of the same ranges, `prepare` builds what a program holds before the call (weights, encoder
object, inputs), `run` makes one pass, `work` and `tolerance` say what the pass cannot do without and how far
two correct implementations may differ.

Fields of a case:
  path     the entry point, see `run`
  model    "base" (12 heads x 64, 12 layers) or "large" (16 heads x 64, 24 layers)
  layers   encoder layers per pass
  batch    sequences
  seq      max_seq of the padded entry points, longest possible sequence of the packed ones
  lengths  how the valid lengths are spread:
             "avg60"   batch 1: round(0.6 seq); else uniform in [2*avg - seq, seq] with avg = 0.6 seq
             "uniform" uniform in [1, seq]
             "long"    uniform in [16, seq]
             "normal"  normal with mean 0.6 seq and deviation 0.21 seq, clipped to [8, seq]
  draw     seed of the lengths: a case's token count is part of the case; the inputs' seed only decides
           which sequence of the batch gets which length, and every value
  gelu     "erf" (what the reference's PyTorch encoder computes) or "tanh" (what its CUDA kernels compute)
  norm32   LayerNorm gamma and beta in fp32 instead of fp16
"""
from __future__ import annotations

import random

import numpy as np
import torch

MODELS = {"base": (12, 12), "large": (16, 24)}   # heads of 64, layers
VOCAB, POSITIONS, TYPES = 30522, 1024, 2         # tables of the embedding front end


def _case(name, path, model, layers, batch, seq, lengths, draw=1, gelu="erf", norm32=False):
    return {"name": name, "path": path, "model": model, "layers": layers, "batch": batch, "seq": seq,
            "lengths": lengths, "draw": draw, "gelu": gelu, "norm32": norm32}


def listed():
    return [
        # the drop-in torch operator of the reference, one layer on a small batch: a call of this kind is made
        # once per layer, so its fixed costs (object, workspace, launches) are paid every time
        _case("op_layer_b16_s64", "op", "base", 1, 16, 64, "uniform"),
        # one short request through a 12-layer model: the smallest forward, latency only
        _case("stack_b1_s64", "stack", "base", 12, 1, 64, "avg60"),
        # one long document
        _case("stack_b1_s1024", "stack", "base", 12, 1, 1024, "avg60"),
        # small batch of sentences with an odd batch and length, tanh GELU and fp32 LayerNorm parameters
        _case("stack_b7_s93_tanh", "stack", "base", 12, 7, 93, "avg60", gelu="tanh", norm32=True),
        # the batch of the reference's published table, short and long sequences
        _case("stack_b16_s128", "stack", "base", 12, 16, 128, "avg60"),
        _case("stack_b16_s512", "stack", "base", 12, 16, 512, "uniform"),
        # BERT-large on a full batch: the largest padded forward
        _case("large_b64_s384", "stack", "large", 24, 64, 384, "normal"),
        # token ids in, pooled sentence vectors out: the whole model front to back
        _case("ids_pool_b32_s128", "ids", "base", 12, 32, 128, "avg60"),
        # causal mask through the general-mask path (every row computed, the whole [B,S,S] mask applied)
        _case("causal_b16_s512", "causal", "base", 12, 16, 512, "uniform"),
        # additive attention bias on an odd sequence length
        _case("bias_b8_s197", "bias", "base", 12, 8, 197, "avg60"),
        # offline throughput over a whole set of sequences held in device memory, packed
        _case("packed_n1024_s1024", "packed", "base", 12, 1024, 1024, "long"),
        # the same from and to pinned host memory, one GPU's share of eight
        _case("host_n128_s1024", "host", "base", 12, 128, 1024, "long"),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng: random.Random):
    path = rng.choice(["op", "stack", "stack", "stack", "stack", "large", "ids", "causal", "bias", "packed", "packed",
                       "host"])
    model, layers, seq = "base", 12, _log_int(rng, 16, 1024)
    if path == "op":
        layers, batch = rng.choice([1, 1, 12]), _log_int(rng, 1, 32)
    elif path == "stack":
        batch = _log_int(rng, 1, 64)
    elif path == "large":
        path, model, layers, batch, seq = "stack", "large", 24, _log_int(rng, 1, 64), _log_int(rng, 16, 512)
    elif path == "ids":
        batch = _log_int(rng, 1, 64)
    elif path == "causal":
        batch = _log_int(rng, 1, 32)
    elif path == "bias":
        batch, seq = _log_int(rng, 1, 16), _log_int(rng, 16, 512)
    elif path == "packed":
        batch, seq = _log_int(rng, 8, 960), _log_int(rng, 32, 1024)
    else:
        batch, seq = _log_int(rng, 16, 128), _log_int(rng, 64, 1024)
    lengths = rng.choice(["uniform", "long"] if path in ("packed", "host") else ["avg60", "uniform", "normal"])
    c = _case("", path, model, layers, batch, seq, lengths, draw=rng.randrange(1, 1 << 20),
              gelu=rng.choice(["erf", "erf", "tanh"]), norm32=rng.choice([False, False, True]))
    if path == "op":
        c["gelu"] = "erf"   # the operator's signature has no such choice
    del c["name"]
    return c


# --------------------------------------------------------------------------------------------- inputs
def _lengths(case):
    """The valid lengths of a case, a function of the case alone."""
    g = torch.Generator().manual_seed(int(case["draw"]))
    B, S = case["batch"], case["seq"]
    kind = case["lengths"]
    if kind == "avg60":
        avg = max(1, int(round(0.6 * S)))
        return torch.tensor([avg]) if B == 1 else torch.randint(max(1, 2 * avg - S), S + 1, (B,), generator=g)
    if kind == "uniform":
        return torch.randint(1, S + 1, (B,), generator=g)
    if kind == "long":
        return torch.randint(min(16, S), S + 1, (B,), generator=g)
    if kind == "normal":
        return torch.clamp(torch.round(torch.randn(B, generator=g) * 0.21 * S + 0.6 * S), min(8, S), S).long()
    raise ValueError(kind)


def _weights(case, dev, g):
    """Layers of random weights: matrices N(0, 0.02) as [in,out], small biases, LayerNorm gamma around 1."""
    H = MODELS[case["model"]][0] * 64
    ln = torch.float32 if case["norm32"] else torch.float16

    def normal(*shape, std=0.02, mean=0.0, dtype=torch.float16):
        return (torch.randn(*shape, generator=g, device=dev) * std + mean).to(dtype).contiguous()

    layers = []
    for _ in range(case["layers"]):
        w = []
        for shape in ((H, 3 * H), (H, H), (H, 4 * H), (4 * H, H)):
            w += [normal(*shape), normal(shape[1])]
            if shape[1] == H:   # the two matrices that a LayerNorm follows
                w += [normal(H, std=0.05, mean=1.0, dtype=ln), normal(H, dtype=ln)]
        layers.append(w)
    return layers


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(int(seed))
    heads = MODELS[case["model"]][0]
    H, B, S, path = heads * 64, case["batch"], case["seq"], case["path"]
    lens = _lengths(case)
    lens = lens[torch.randperm(B, generator=torch.Generator().manual_seed(int(seed)))]
    layers = _weights(case, dev, g)
    st = {"path": path, "heads": heads, "layers": layers}

    def activations(*shape):
        return torch.randn(*shape, generator=g, device=dev).half()

    if path == "op":
        from bytetransformer_b200 import build
        torch.ops.load_library(build.THS_LIB)
        st["op"] = torch.ops.ByteTransformer.BertTransformer
    else:
        from bytetransformer_b200.encoder import Encoder
        st["enc"] = Encoder(heads, 64, layers, gelu=case["gelu"])
    if path in ("packed", "host"):
        from bytetransformer_b200.runner import PackedRunner
        st["runner"] = r = PackedRunner(st["enc"], lens.numpy(), np.arange(B), min_batches=1 if path == "packed" else 4)
        st["x"] = [activations(mb.tokens, H) for mb in r.batches]
        if path == "host":
            st["x"] = [x.cpu().pin_memory() for x in st["x"]]
            st["out"] = [torch.empty(x.shape, dtype=x.dtype, pin_memory=True) for x in st["x"]]
        else:
            st["out"] = [torch.empty_like(x) for x in st["x"]]
        return st
    valid = torch.arange(S)[None, :] < lens[:, None]
    mask = valid[:, None, :].expand(B, S, S)
    if path == "causal":
        mask = mask & torch.ones(S, S, dtype=torch.bool).tril()
    st["mask"] = mask.to(dev).half().contiguous()
    if path == "ids":
        from bytetransformer_b200.encoder import EmbeddingWeights
        ln = torch.float32 if case["norm32"] else torch.float16
        table = [(torch.randn(n, H, generator=g, device=dev) * 0.02).half() for n in (VOCAB, POSITIONS, TYPES)]
        st["emb"] = EmbeddingWeights(*table, torch.ones(H, device=dev, dtype=ln), torch.zeros(H, device=dev, dtype=ln))
        st["ids"] = torch.randint(0, VOCAB, (B, S), generator=g, device=dev, dtype=torch.int32)
        st["types"] = torch.randint(0, TYPES, (B, S), generator=g, device=dev, dtype=torch.int32)
        st["pool"] = [(torch.randn(H, H, generator=g, device=dev) * 0.02).half(), activations(H) * 0.02]
    else:
        st["x"] = activations(B, S, H)
    if path == "bias":
        st["bias"] = activations(heads, S, S)
    return st


# ------------------------------------------------------------------------------------------- one pass
def run(st):
    path = st["path"]
    if path == "stack":      # padded batch in, padded batch out, all layers in one call
        return st["enc"].forward(st["x"], st["mask"])
    if path == "op":         # the reference's own loop over its operator
        x = st["x"]
        for w in st["layers"]:
            x = st["op"](st["heads"], 64, *w, x, st["mask"], True, True)
        return x
    if path == "ids":
        y = st["enc"].forward_ids(st["emb"], st["ids"], st["mask"], type_ids=st["types"])
        from bytetransformer_b200.encoder import pooler
        return y, pooler(y, *st["pool"])
    if path == "causal":
        return st["enc"].forward_general(st["x"], st["mask"])
    if path == "bias":
        return st["enc"].forward_general(st["x"], st["mask"], attention_bias=st["bias"])
    if path == "packed":
        st["runner"].run_device(st["x"], st["out"])
        return st["out"]
    st["runner"].run_host(st["x"], st["out"])
    return st["out"]


# --------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Matrix products over the rows that have to be computed, attention over the pairs that the mask leaves
    (both products), and each input, weight and output once.  The packed paths compute the valid rows; the
    general-mask paths are asked for every row, a right-padded or causal mask leaving each its own keys."""
    heads = MODELS[case["model"]][0]
    H, B, S, nl, path = heads * 64, case["batch"], case["seq"], case["layers"], case["path"]
    l = _lengths(case).numpy().astype(np.float64)
    if path in ("causal", "bias"):
        rows = float(B * S)
        pairs = float((l * S).sum()) if path == "bias" else float((l * (l + 1) / 2 + (S - l) * l).sum())
    else:
        rows, pairs = float(l.sum()), float((l * l).sum())
    flops = nl * (24.0 * rows * H * H + 4.0 * H * pairs)
    nbytes = nl * (24.0 * H * H + 26.0 * H)                                # weights
    if path in ("packed", "host"):
        nbytes += 4.0 * rows * H + 4.0 * (B + 1)                           # packed rows in and out, offsets
    else:
        nbytes += 2.0 * B * S * H + (2.0 * rows * H if path != "ids" else 0.0)   # padded output, input rows
        nbytes += 2.0 * B * S * S if path in ("causal", "bias") else 2.0 * B * S  # mask: all of it, or its first rows
    if path == "bias":
        nbytes += 2.0 * heads * S * S
    if path == "ids":
        nbytes += 8.0 * rows + 2.0 * min(rows, float(VOCAB)) * H + 2.0 * (S + TYPES) * H + 2.0 * H * H + 2.0 * B * H
        flops += 2.0 * B * H * H
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """fp16 activations between the kernels, fp32 sums.  Measured against the same forward in fp32 throughout: 3.0e-4
    (largest single value 1.5e-3) for one layer, 1.0e-3 to 1.15e-3 (5e-3 to 1.1e-2) for 12 and 24 layers, where
    LayerNorm keeps the error from growing with depth; four times that is allowed."""
    return {"rel": 4e-3, "max": 4e-2} if case["layers"] > 1 else {"rel": 1.3e-3, "max": 6e-3}
