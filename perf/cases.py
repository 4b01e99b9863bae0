"""Performance cases of the quantized KV cache: what they are, how their inputs are made, how one pass runs.

Five kinds of call, each through the public entry points that a model integration uses:

  decode     one token's attention over a filled layer (``mu_zero_decode_attention_forward``)
  generate   a layer's share of a short generation: prompt block into a new cache, then decode steps
             (``MuZeroCache.update`` + ``mu_zero_decode_step_forward``: append, flush when due, attention)
  prefill    a prompt block into a new cache: alpha choice, quantization, residual window (``MuZeroCache.update``)
  dense      the layer's keys and values back as ordinary tensors, what a model without the fused decode path
             attends to (``MuZeroCache.__getitem__``)
  roundtrip  quantize and dequantize a key / value block (``roundtrip``), the quality tool

Sizes: 8 kv heads, 32 query heads, head_dim 128, group 64 and a residual window of 128 tokens are the benchmark's
attention shape; contexts of 2048 to 32768, batches of 32 to 64 and the 131072-token batch of 8 are its sweeps.
Other head ratios, head_dim 64, groups of 32 and 128, and 1, 3, 7 and 8 bits are what the tests cover.
"""
import math

import torch

import muzero_b200 as mz

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, kind, batch, tokens, bits, **kw):
    c = {"name": name, "kind": kind, "batch": batch, "tokens": tokens, "bits": bits, "group": 64, "kv_heads": 8, "q_heads": 32,
         "head_dim": 128, "dtype": "bf16", "mask": False, "steps": 0}
    c.update(kw)
    return c


def listed():
    return [
        # a chat turn of one user: a short context, where launches and host work are all there is
        _case("decode_single", "decode", 1, 500, 4),
        # the benchmark's batch of 64 sequences at 4096 tokens and the residual window
        _case("decode_batch", "decode", 64, 4224, 4),
        # long documents: the 131072-token stress batch, with the smallest codes that are served
        _case("decode_long_2bit", "decode", 8, 131072, 2),
        # the near-lossless setting on a half-precision model
        _case("decode_8bit", "decode", 16, 4000, 8, dtype="fp16"),
        # prompts of unlike lengths, left-padded under an additive mask, on a model with 8 query heads per kv head
        _case("decode_padded", "decode", 6, 1777, 4, q_heads=64, mask=True),
        # a small model: head_dim 64
        _case("decode_head64", "decode", 16, 2050, 4, head_dim=64),
        # generation for two users
        _case("generate_small", "generate", 2, 500, 4, steps=32),
        # a batch job with 3-bit codes: alpha statistics in the prefill, one flush among the steps
        _case("generate_3bit", "generate", 24, 1537, 3, steps=32),
        # one prompt, as a chat front end sends it
        _case("prefill_single", "prefill", 1, 2047, 4),
        # a batch of long prompts with data-dependent alphas
        _case("prefill_batch_2bit", "prefill", 16, 4096, 2),
        # a model family without the fused decode path: the whole cache as dense keys and values
        _case("dense_batch", "dense", 8, 4224, 4),
        # quality evaluation of a setting on captured keys and values
        _case("roundtrip", "roundtrip", 2, 2048, 4),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["decode", "generate", "prefill", "dense", "roundtrip"], [6, 2, 3, 1, 1])[0]
    bits = rng.choices([4, 2, 8, 3, 1, 7], [8, 4, 3, 3, 1, 1])[0]
    head_dim = rng.choices([128, 64], [5, 1])[0]
    group = rng.choices([64, 32, 128], [6, 1, 1])[0]
    group = min(group, head_dim)
    kv_heads = rng.choice([2, 4, 8, 8])
    q_heads = kv_heads * rng.choices([1, 2, 4, 8], [1, 1, 4, 2])[0]
    batch = _log_uniform(rng, 1, 64)
    # tokens over all (batch, kv head) pairs stay below the batch benchmark's for decode, the batch prefill's otherwise
    most = (64 * 8 * 4224 if kind == "decode" else 16 * 8 * 4096) // (batch * kv_heads)
    tokens = _log_uniform(rng, 200, max(400, min(most, 131072 if kind == "decode" else 16384)))
    if kind == "roundtrip":
        tokens = -(-tokens // group) * group        # it takes whole key groups
    return {"kind": kind, "batch": batch, "tokens": tokens, "bits": bits, "group": group, "kv_heads": kv_heads, "q_heads": q_heads,
            "head_dim": head_dim, "dtype": rng.choices(["bf16", "fp16"], [3, 1])[0],
            "mask": kind == "decode" and rng.random() < 0.25, "steps": rng.randint(8, 32) if kind == "generate" else 0}


class _Module:
    """The part of a model's attention module that the decode hooks read."""

    def __init__(self, groups):
        self.num_key_value_groups = groups


def _key_value_block(c, tokens, gen):
    """Keys and values [B,KVH,S,D] in the layout of a model's projections ([B,S,KVH,D] underneath): values ~ N(0,1),
    keys ~ N(0,1) with log-normal channel scales."""
    shape, dt = (c["batch"], tokens, c["kv_heads"], c["head_dim"]), _DTYPES[c["dtype"]]
    chan = torch.exp(torch.randn(c["head_dim"], device="cuda", generator=gen))
    v = torch.randn(shape, device="cuda", generator=gen, dtype=dt)
    k = torch.randn(shape, device="cuda", generator=gen, dtype=dt).mul_(chan.to(dt))
    return k.transpose(1, 2), v.transpose(1, 2), chan


def _config(c):
    return mz.MuZeroConfig(bits=c["bits"], q_group_size=c["group"], residual_length=128)


def _filled_cache(c, k, v):
    cache = mz.MuZeroCache(_config(c))
    cache.update(k, v, 0, {"materialize_full_kv": False})
    return cache


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[c["dtype"]]
    k, v, chan = _key_value_block(c, c["tokens"], gen)
    s = {"case": c, "scaling": c["head_dim"] ** -0.5, "module": _Module(c["q_heads"] // c["kv_heads"])}
    if c["kind"] == "decode":
        s["cache"] = _filled_cache(c, k, v)
        s["query"] = torch.randn(c["batch"], 1, c["q_heads"], c["head_dim"], device="cuda", generator=gen, dtype=dt).transpose(1, 2)
        s["mask"] = None
        if c["mask"]:       # left padding of up to half the context, the first sequence unpadded
            pad = (torch.rand(c["batch"], device="cuda", generator=gen) * (c["tokens"] // 2)).long()
            pad[0] = 0
            dead = torch.arange(c["tokens"], device="cuda")[None, :] < pad[:, None]
            s["mask"] = torch.zeros(c["batch"], 1, 1, c["tokens"], device="cuda", dtype=dt).masked_fill_(
                dead[:, None, None, :], torch.finfo(dt).min)
    elif c["kind"] == "generate":
        s["k"], s["v"] = k, v
        n, b = c["steps"], c["batch"]
        ks = torch.randn(n, b, 1, c["kv_heads"], c["head_dim"], device="cuda", generator=gen, dtype=dt).mul_(chan.to(dt))
        vs = torch.randn(n, b, 1, c["kv_heads"], c["head_dim"], device="cuda", generator=gen, dtype=dt)
        qs = torch.randn(n, b, 1, c["q_heads"], c["head_dim"], device="cuda", generator=gen, dtype=dt)
        s["steps"] = [(ks[i].transpose(1, 2), vs[i].transpose(1, 2), qs[i].transpose(1, 2)) for i in range(n)]
    elif c["kind"] == "dense":
        s["cache"] = _filled_cache(c, k, v)
    else:
        s["k"], s["v"] = k, v
    return s


def _layer_state(layer):
    return {"packed_k": layer._packed_key_q, "k_mn": layer._key_mn, "k_scale": layer._key_scale,
            "packed_v": layer._packed_value_q, "v_mn": layer._value_mn, "v_scale": layer._value_scale,
            "keys": layer.keys, "values": layer.values}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "decode":
        attn = state["cache"].get_attention_state(0)
        return mz.mu_zero_decode_attention_forward(state["module"], state["query"], state["mask"], state["scaling"], attn)[0]
    if kind == "generate":
        cache = _filled_cache(c, state["k"], state["v"])
        layer, outs = cache.layers[0], []
        for k, v, q in state["steps"]:
            outs.append(mz.cache.attention.mu_zero_decode_step_forward(state["module"], layer, k, v, q, None, state["scaling"])[0])
        return {"out": outs, **_layer_state(layer)}
    if kind == "prefill":
        return _layer_state(_filled_cache(c, state["k"], state["v"]).layers[0])
    if kind == "dense":
        k, v = state["cache"][0]
        return k[0], v[0]
    return mz.roundtrip(state["k"], state["v"], bits=c["bits"], q_group_size=c["group"])


def _split(c, tokens):
    """(quantized, residual) tokens after a prompt of `tokens`: whole groups beyond the residual window are quantized."""
    q = max(tokens - 128, 0) // c["group"] * c["group"]
    return q, tokens - q


def _store_bytes(c, quantized):
    """Packed codes and fp16 (min, range) of keys and values, all pairs."""
    d, g = c["head_dim"], c["group"]
    per_token = 2 * d * c["bits"] / 8 + 2 * 4 * d / g
    return c["batch"] * c["kv_heads"] * quantized * per_token


def _dense_bytes(c, tokens):
    return c["batch"] * c["kv_heads"] * tokens * c["head_dim"] * 2 * 2


def _decode_work(c, tokens):
    q, r = _split(c, tokens)
    heads = c["batch"] * c["q_heads"] * c["head_dim"]
    nbytes = _store_bytes(c, q) + _dense_bytes(c, r) + 2 * 2 * heads + (2 * c["batch"] * tokens if c["mask"] else 0)
    return nbytes, 4 * heads * tokens


def work(case):
    c, n = case, case["tokens"]
    q, r = _split(c, n)
    values = 2 * c["batch"] * c["kv_heads"] * n * c["head_dim"]
    if c["kind"] == "decode":
        nbytes, flops = _decode_work(c, n)
    elif c["kind"] == "prefill":
        nbytes, flops = _dense_bytes(c, n) + _store_bytes(c, q) + _dense_bytes(c, r), 10 * values
    elif c["kind"] == "generate":
        nbytes, flops = _dense_bytes(c, n) + _store_bytes(c, q) + _dense_bytes(c, r), 10 * values
        for i in range(c["steps"]):
            b, f = _decode_work(c, n + i + 1)
            nbytes, flops = nbytes + b + 2 * _dense_bytes(c, 1), flops + f
    elif c["kind"] == "dense":
        nbytes, flops = _store_bytes(c, q) + _dense_bytes(c, r) + _dense_bytes(c, n), 4 * values
    else:
        nbytes, flops = 2 * _dense_bytes(c, n), 14 * values
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # attention outputs are bf16 / fp16; codes, metadata and dequantized values are the same bits everywhere
    if case["kind"] == "decode":
        return {"rel": 1e-2}
    if case["kind"] == "generate":
        return {"rel": 1e-2, "differ": 0.0}
    return "exact"
