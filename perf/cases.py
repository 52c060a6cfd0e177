"""Performance cases of the FP8 block-scaled MoE layer: the calls a serving or training program makes, over
the range of batch sizes, expert counts and options the layer takes, with inputs of the distributions the
layer's generators (`gen.py`) stand for.

A case is a dict of plain values:

  tokens                 T, rows of the batch
  experts, offset        local experts of this GPU (32 = one shard of an eight-GPU job, 256 = all) and the first one
  layers                 MoE layers a pass runs one after the other through ONE handle, as a model does: each
                         layer has its own weights, router and activations, the workspace is shared
  entry                  "fp8": quantised activations in hand; "bf16": quantise-on-entry, then the layer;
                         "host": the per-call tensors live in pinned host memory; "dropin": the module-level
                         `run(...)` with the reference's eleven arguments
  skew                   Zipf-like expert popularity instead of near-uniform routing
  prune, exact_silu      the layer's two numerical options (defaults: on, off)
  hidden, inter, top_k, n_group, topk_group    the layer's shape
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

import __graft_entry__ as entry

NE = 256
RSF = 2.5
REFERENCE_SHAPE = dict(hidden=7168, inter=2048, top_k=8, n_group=8, topk_group=4)
# other shapes the layer is built for, as its shape tests and documents use them
OTHER_SHAPES = (
    dict(hidden=4096, inter=1536, top_k=8, n_group=1, topk_group=1),
    dict(hidden=2048, inter=1024, top_k=6, n_group=1, topk_group=1),
    dict(hidden=7168, inter=1920, top_k=8, n_group=8, topk_group=4),
)


def _case(name=None, **kw):
    c = dict(tokens=1, experts=32, offset=0, layers=1, entry="fp8", skew=False, prune=True, exact_silu=False)
    c.update(REFERENCE_SHAPE)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one decode token through four consecutive MoE layers of a model, by the drop-in operator: latency,
        # launches and host work
        _case("decode_t1_4layers", tokens=1, layers=4, entry="dropin"),
        # a decode step of eight sequences on one GPU that holds all experts: about fifty experts' weights stream
        _case("decode_t8_e256", tokens=8, experts=256),
        # a small batch on one shard of an eight-GPU job
        _case("batch_t16", tokens=16),
        # a decode batch of odd size, activations quantised on entry
        _case("batch_t57_bf16", tokens=57, offset=96, entry="bf16"),
        # a decode batch of 128 sequences on one GPU with all experts: every expert's weights are read for a few rows
        _case("batch_t128_e256", tokens=128, experts=256),
        # a short odd prefill by the layer's exact definition (exact SiLU, every selected expert kept)
        _case("prefill_t901_exact", tokens=901, offset=160, prune=False, exact_silu=True),
        # chunked prefill of 1024 tokens, two layers of the model through one workspace
        _case("prefill_t1024_2layers", tokens=1024, layers=2),
        # a host-resident caller: pinned activations in, pinned output back, one blocking call
        _case("host_t2048", tokens=2048, entry="host"),
        # a ragged prefill on a quarter of the experts (four-GPU job), bf16 activations
        _case("prefill_t4099_e64_bf16", tokens=4099, experts=64, offset=64, entry="bf16"),
        # the headline batch: 12288 tokens, all 256 experts on one GPU
        _case("prefill_t12288_e256", tokens=12288, experts=256),
        # the longest batch with a skewed router, half of the experts (two-GPU job): hot experts, long tails
        _case("skew_t16384_e128", tokens=16384, experts=128, offset=64, skew=True),
        # a model of another shape, half of its experts on this GPU
        _case("shape_4096x1536_t3000", tokens=3000, experts=128, offset=128, **OTHER_SHAPES[0]),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    experts = rng.choice((32, 32, 32, 64, 128, 256))
    tokens = _log_int(rng, 1, 12288 if experts == 256 else 16384)
    shape = REFERENCE_SHAPE if rng.random() < 0.8 else rng.choice(OTHER_SHAPES)
    layers = 1
    if experts <= 64 and tokens <= 2048:
        layers = rng.choice((1, 1, 2, 4) if experts == 32 else (1, 1, 2))
    kinds = ["fp8", "fp8", "bf16"]
    if tokens <= 4096 and layers == 1:
        kinds.append("host")
    # the drop-in operator's handle remembers weight scales by address for batches of more than eight tokens, so
    # here, where weights come and go, it serves the decode sizes only
    if tokens <= 8 and shape is REFERENCE_SHAPE:
        kinds += ["dropin", "dropin"]
    kind = rng.choice(kinds)
    plain = kind == "dropin"
    return _case(tokens=tokens, experts=experts, offset=32 * rng.randrange((NE - experts) // 32 + 1), layers=layers,
                 entry=kind, skew=rng.random() < 0.25, prune=plain or rng.random() < 0.8,
                 exact_silu=not plain and rng.random() < 0.2, **shape)


# ------------------------------------------------------------------------------------------------ inputs
def _package():
    moe = entry.load_package()
    from fp8_moe_dev_b200 import gen
    return moe, gen


def _seed(seed, *what):
    """A seed for one tensor of one layer: other cases' seeds give other tensors throughout."""
    return zlib.crc32(repr((int(seed),) + what).encode()) & 0x7FFFFFFF


def _one_layer(c, seed, i, gen):
    """Router outputs, activations, weights and the output buffer of layer `i`."""
    T, H, inter = c["tokens"], c["hidden"], c["inter"]
    logits, bias = gen.make_routing(T, _seed(seed, i, "routing"), c["skew"], device="cuda",
                                    skew_seed=_seed(seed, i, "skew"))
    w1, s1, w2, s2 = gen.make_shard(c["offset"], c["experts"], base_seed=_seed(seed, i, "weights"), device="cuda",
                                    hidden=H, inter=inter)
    t = dict(logits=logits, bias=bias, w1=w1, s1=s1, w2=w2, s2=s2)
    g = torch.Generator(device="cuda")
    g.manual_seed(_seed(seed, i, "hidden"))
    x = torch.randn(T, H, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    if c["entry"] == "bf16":
        t["x"] = x
        t["q"] = torch.empty(T, H, dtype=torch.float8_e4m3fn, device="cuda")
        t["scale"] = torch.empty(H // 128, T, dtype=torch.float32, device="cuda")
    else:
        t["q"], t["scale"] = gen.quantize_rows_1x128(x)
    t["out"] = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    if c["entry"] == "host":
        for k in ("logits", "q", "scale", "out"):
            t[k] = t[k].cpu().pin_memory()
    return t


def prepare(case, seed):
    moe, gen = _package()
    s = dict(case=case, moe=moe, layers=[_one_layer(case, seed, i, gen) for i in range(case["layers"])])
    if case["entry"] != "dropin":
        h = moe.MoeLayer(case["tokens"], case["experts"], hidden=case["hidden"], intermediate=case["inter"],
                         top_k=case["top_k"], n_group=case["n_group"], topk_group=case["topk_group"])
        if not case["prune"]:
            h.set_reference_pruning(False)
        if case["exact_silu"]:
            h.set_exact_silu(True)
        s["handle"] = h
    return s


def run(state):
    c, outs = state["case"], []
    for t in state["layers"]:
        weights = (t["w1"], t["s1"], t["w2"], t["s2"], c["offset"], RSF)
        if c["entry"] == "dropin":
            state["moe"].run(t["logits"], t["bias"], t["q"], t["scale"], *weights, t["out"])
        elif c["entry"] == "host":
            state["handle"].run_host(t["logits"], t["bias"], t["q"], t["scale"], *weights, t["out"])
        else:
            if c["entry"] == "bf16":
                state["handle"].quantize_hidden(t["x"], t["q"], t["scale"])
                # the codes as bytes: they are whole values, compared as such
                outs += [t["q"].view(torch.uint8), t["scale"]]
            state["handle"].run(t["logits"], t["bias"], t["q"], t["scale"], *weights, t["out"])
        outs.append(t["out"])
    return outs


# ------------------------------------------------------------------------------------------------ what it costs
def _routed(c):
    """Expected (rows, experts with a row, tokens with a row) of one layer: the mean over a few samples of the
    routing distribution, more of them the fewer tokens there are or the more a single expert weighs."""
    rng = np.random.Generator(np.random.PCG64(12))
    samples = max(4 if c["skew"] else 1, 512 // c["tokens"])
    return np.mean([_routed_once(c, rng) for _ in range(samples)], axis=0)


def _routed_once(c, rng):
    """One sample: biased sigmoid scores, groups by the sum of their two best, top experts, then (option `prune`,
    batches of 32 tokens or more) at most three experts per 32-expert shard and token, in the longest batches a
    third one only above its share."""
    T = c["tokens"]
    logits = rng.standard_normal((T, NE), dtype=np.float32)
    if c["skew"]:
        logits += 1.5 * np.log(1.0 / (rng.permutation(NE) + 1)).astype(np.float32)[None, :]
    score = 1.0 / (1.0 + np.exp(-logits))
    biased = score + 0.1 * rng.standard_normal(NE, dtype=np.float32)[None, :]
    groups = np.sort(biased.reshape(T, c["n_group"], -1), axis=2)[:, :, -2:].sum(axis=2)
    kept = np.argsort(-groups, axis=1)[:, :c["topk_group"]]
    live = np.zeros((T, c["n_group"]), dtype=bool)
    np.put_along_axis(live, kept, True, axis=1)
    masked = np.where(np.repeat(live, NE // c["n_group"], axis=1), biased, -np.inf)
    idx = np.argsort(-masked, axis=1)[:, :c["top_k"]]
    w = np.zeros((T, NE), dtype=np.float32)
    np.put_along_axis(w, idx, np.take_along_axis(score, idx, axis=1), axis=1)
    if c["prune"] and T >= 32:
        shards = w.reshape(T, NE // 32, 32)
        order = np.sort(shards, axis=2)
        third, total = order[:, :, -3], shards.sum(axis=2)
        least = third
        if T >= 10000:
            least = np.where(third <= (0.34 if T < 13000 else 0.30) * total, order[:, :, -2], third)
        w = np.where(shards >= np.maximum(least, 1e-30)[:, :, None], shards, 0.0).reshape(T, NE)
    local = w[:, c["offset"]:c["offset"] + c["experts"]] > 0
    return int(local.sum()), int(local.any(axis=0).sum()), int(local.any(axis=1).sum())


def work(case):
    """What one pass cannot do without: the weights of the experts that have a row, once; the routing inputs; the
    activations of the tokens with a row; the output.  Two GEMMs' multiply-adds per routed row."""
    T, H, inter = case["tokens"], case["hidden"], case["inter"]
    rows, experts, tokens = _routed(case)
    weights = experts * (3 * H * inter + 4 * 3 * H * inter / (128 * 128))
    acts = tokens * (H + 4 * H // 128)
    if case["entry"] == "bf16":
        acts = T * (2 * H + H + 4 * H // 128)   # every row read, its codes and scales are results
    one = weights + acts + T * NE * 4 + NE * 2 + T * H * 2
    return {"bytes": float(case["layers"] * one), "flops": float(case["layers"] * rows * 6 * H * inter)}


def tolerance(case):
    # bf16 results whose intermediate activations pass through bf16 and e4m3: another order of the fp32 sums moves
    # some of those to the neighbouring code.  The codes of the quantise-on-entry form are whole values: none differ.
    return {"rel": 1e-2, "max": 0.2, "differ": 0.0}
