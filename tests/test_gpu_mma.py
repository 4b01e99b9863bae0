"""GPU: the tensor-core decode kernel at the edges of its tiles, widths and head sets, in its cluster and flat forms."""
from contextlib import contextmanager

import pytest
import torch

from test_gpu_attention import SPLIT_TOL, check_output

pytestmark = pytest.mark.gpu


@contextmanager
def kernel(which):
    """Decode calls inside go to one kernel (4: the tcgen05 kernel for all that it serves)."""
    from muzero_b200.kernels._cabi import load_library
    lib = load_library()
    before = lib.mz_debug_force_kernel(which)
    try:
        yield
    finally:
        lib.mz_debug_force_kernel(before)


@pytest.mark.parametrize("gqa,S,residual", [(1, 65, 64), (3, 300, 64), (4, 129 + 128, 128), (5, 450, 64), (8, 1000, 128), (7, 40, 64)])
@pytest.mark.parametrize("bits,D,group", [(1, 64, 32), (2, 128, 128), (3, 128, 32), (3, 64, 64), (4, 64, 64), (4, 128, 128), (4, 128, 64),
                                          (5, 128, 64), (7, 64, 32), (8, 64, 64), (8, 128, 128)])
def test_widths_groups_heads(oracle, bits, D, group, gqa, S, residual):
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    residual = max(residual, group)
    k, v, q = oracle.synth_kv(2, 2, S + 3, D, 2 * gqa, seed=bits * 7 + gqa)
    k[:, :, :, :3] += 4.0        # rows that do not straddle zero, and symmetric ones (their zero code is a tie)
    v[0] -= 3.0
    k[0, 0, 0::2, 5], k[0, 0, 1::2, 5] = 1.5, -1.5
    ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=residual, alpha_key=2.0, alpha_value=4.0)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=residual, alpha_key=2.0, alpha_value=4.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    ref.append(k[:, :, :S].contiguous(), v[:, :, :S].contiguous())
    layer.update(k[:, :, :S].cuda().contiguous(), v[:, :, :S].cuda().contiguous(), {"materialize_full_kv": False})
    for i in range(S, S + 3):
        ref.append(k[:, :, i:i + 1].contiguous(), v[:, :, i:i + 1].contiguous())
        got = layer.decode_step(k[:, :, i:i + 1].cuda(), v[:, :, i:i + 1].cuda(), q.cuda(), D ** -0.5)
    want = oracle.decode_attention_oracle(q, ref, D ** -0.5, gqa, compute_dtype=torch.float32)
    o32 = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32)
    check_output(o32, got, want)
    assert torch.equal(layer.keys.cpu(), ref.keys) and torch.equal(layer.values.cpu(), ref.values)
    for splits in (1, 3):
        assert (decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32, splits=splits) - o32).abs().max().item() < SPLIT_TOL
    mask = torch.zeros(2, 1, 1, S + 3).masked_fill_(torch.rand(2, 1, 1, S + 3, generator=torch.Generator().manual_seed(1)) < 0.3, -1e30)
    want = oracle.decode_attention_oracle(q, ref, D ** -0.5, gqa, mask=mask, compute_dtype=torch.float32)
    check_output(decode_attention(layer, q.cuda(), D ** -0.5, mask.cuda(), out_dtype=torch.float32),
                 decode_attention(layer, q.cuda(), D ** -0.5, mask.cuda()), want)


def attention64(oracle, ref, q, scaling, mask=None):
    """Attention over the oracle's dequantized store and window, evaluated in 64 bits: [B,1,H,D]."""
    k = torch.cat(([ref.key_prefix(torch.float32)] if ref.packed_k is not None else []) + [ref.keys.float()], dim=2).double()
    v = torch.cat(([ref.value_prefix(torch.float32)] if ref.packed_v is not None else []) + [ref.values.float()], dim=2).double()
    b, h, _, d = q.shape
    logits = torch.matmul(q.double().reshape(b, k.shape[1], -1, d), k.transpose(2, 3)) * scaling
    if mask is not None:
        logits = logits + mask.double()
    return torch.matmul(torch.softmax(logits, dim=-1), v).reshape(b, 1, h, d)


def relative_error(got, want):
    return ((got.double().cpu() - want).norm() / want.norm()).item()


# About twenty fp32 roundings (2^-24 each) lie between the inputs and an output: the dequantizer's, the product and sum of
# the logits (relative to a logit of up to about 8), exponential, products and sums of the values.  Sums over tokens
# average them.  2e-6 is the plain sum of the twenty, times 1.6.
FP32_ERROR = 2e-6
# channels a thousandth of their group's range: the group's dequantized values round relative to the range
SHARED_GROUP_ERROR = 1e3 * FP32_ERROR


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits,D,group,gqa", [(1, 128, 64, 8), (2, 128, 128, 4), (2, 64, 64, 3), (3, 128, 64, 4), (3, 64, 32, 8), (4, 128, 64, 8),
                                              (4, 128, 32, 4), (4, 64, 64, 1), (5, 64, 64, 4), (8, 128, 64, 8), (8, 64, 32, 2)])
def test_error_against_64_bits(oracle, bits, D, group, gqa, dtype):
    """The general tensor-core kernel (cluster mode and flat cut) has the error of an fp32 evaluation; the residual window
    alone as well."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    for S in (100, 900):
        k, v, q = oracle.synth_kv(2, 2, S, D, 2 * gqa, seed=bits + D, dtype=dtype)
        ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=128, alpha_key=2.0, alpha_value=4.0)
        ref.append(k, v)
        cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=128, alpha_key=2.0, alpha_value=4.0)
        cfg.bits = bits
        layer = mz.MuZeroCacheLayer(cfg)
        layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
        want = attention64(oracle, ref, q, D ** -0.5)
        for splits in (0, 5):
            got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32, splits=splits)
            assert relative_error(got, want) <= FP32_ERROR, (S, splits)


@pytest.mark.parametrize("vs,ks,qs,meta", [(1e-4, 1.0, 1.0, torch.float16), (1e-6, 1.0, 1.0, torch.float32), (1e5, 1.0, 1.0, torch.float32),
                                           (1e5, 1.0, 1.0, torch.bfloat16), (1.0, 1e-4, 1e4, torch.float16), (1.0, 1e5, 1e-5, torch.float32)])
@pytest.mark.parametrize("bits,D,group,gqa", [(1, 128, 128, 2), (3, 128, 64, 4), (4, 128, 64, 8), (4, 64, 32, 4), (8, 64, 64, 4)])
def test_error_at_any_scale(oracle, bits, D, group, gqa, vs, ks, qs, meta):
    """Ranges far from 1: below fp16's smallest normal value times 2^11, above its largest; value groups of unlike scale."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = (t.float() for t in oracle.synth_kv(2, 2, 700, D, 2 * gqa, seed=bits))
    v[..., :32] *= 1e-3
    k, v, q = ((t * f).to(torch.bfloat16) for t, f in ((k, ks), (v, vs), (q, qs)))
    ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=128, meta_dtype=meta, alpha_key=2.0, alpha_value=2.0)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=128, amax_dtype=str(meta)[6:], alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    want = attention64(oracle, ref, q, D ** -0.5)
    for splits in (0, 3):
        got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32, splits=splits)
        assert bool(torch.isfinite(got).all())
        for part in (slice(0, 32), slice(32, D)):
            assert relative_error(got[..., part], want[..., part]) <= (FP32_ERROR if part.start or group == 32 else SHARED_GROUP_ERROR)


@pytest.mark.parametrize("bits,D,group,gqa,B,S", [(4, 128, 64, 8, 12, 1777), (3, 128, 32, 8, 10, 725), (1, 128, 128, 2, 12, 1777), (8, 64, 32, 4, 18, 601),
                                                  (4, 128, 32, 2, 16, 800), (4, 128, 64, 4, 18, 289), (2, 128, 64, 4, 1, 11213), (5, 128, 64, 1, 8, 1500)])
def test_clusters_whose_warps_take_several_tiles(oracle, bits, D, group, gqa, B, S):
    """Up to 148 pairs with more tiles than the pair's cluster has warps, on both sides of the choice between a cluster and an
    even cut; the forced cut of the same call gives the same values."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(B, 8, S, D, 8 * gqa, seed=bits + S)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=128, alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    mask = torch.zeros(B, 1, 1, S)
    mask[B - 1, ..., : S // 2] = torch.finfo(torch.bfloat16).min
    got = decode_attention(layer, q.cuda(), D ** -0.5, mask.cuda(), out_dtype=torch.float32).cpu()
    cut = decode_attention(layer, q.cuda(), D ** -0.5, mask.cuda(), out_dtype=torch.float32, splits=2).cpu()
    unrolled = group == 64 and D == 128 and bits in (2, 4) and gqa <= 4         # its cut has the error pinned below
    assert relative_error(got, cut.double()) <= (1.2e-4 if unrolled else 2 * FP32_ERROR)
    for b in {0, B - 1}:
        ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=128, alpha_key=2.0, alpha_value=2.0)
        ref.append(k[b:b + 1], v[b:b + 1])
        want = attention64(oracle, ref, q[b:b + 1], D ** -0.5, mask[b:b + 1])
        assert relative_error(got[b:b + 1], want) <= (1.2e-4 if unrolled else FP32_ERROR)


@pytest.mark.parametrize("bits,D,group,gqa", [(3, 128, 64, 4), (4, 64, 32, 8), (8, 128, 64, 8)])
def test_an_infinite_range_stays_in_its_group(oracle, bits, D, group, gqa):
    """A value range that overflowed fp16 metadata makes its own channels non-finite, as the dequantizer does, and no others."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(2, 2, 500, D, 2 * gqa, seed=bits)
    ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=128, alpha_key=2.0, alpha_value=2.0)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=128, alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    layer._value_scale[0, 1, 5, 1] = float("inf")
    got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32).cpu()
    want = attention64(oracle, ref, q, D ** -0.5)
    hit = torch.zeros(got.shape, dtype=torch.bool)
    hit[0, :, gqa:, group:2 * group] = True
    assert not bool(torch.isfinite(got[hit]).any()) and relative_error(got[~hit], want[~hit]) <= FP32_ERROR


def unlike_tokens(oracle, kind, batch, kv_heads, tokens, head_dim, gqa, seed):
    """Keys, values and queries whose largest factors do not meet in one product.  sink: one token dominates by 8 or 12 nats and has values a
    hundredth or a thousandth of the others' (early: in the first step of a range; late: behind others).  outlier: a key channel a thousand or
    ten thousand times the others' under a query as much smaller.  spread: tokens' values over a factor of 400."""
    k, v, q = (t.float() for t in oracle.synth_kv(batch, kv_heads, tokens, head_dim, kv_heads * gqa, seed=seed))
    gen = torch.Generator().manual_seed(seed)
    if kind.startswith("sink"):
        nats = 8.0 if "8" in kind else 12.0
        at = tokens - 300 if kind.endswith("late") else 5
        base = torch.randn(1, kv_heads, 1, 1, head_dim, generator=gen).sign()
        q = (base + 0.3 * torch.randn(batch, kv_heads, gqa, 1, head_dim, generator=gen)).reshape(batch, kv_heads * gqa, 1, head_dim)
        k = 0.3 * torch.randn(batch, kv_heads, tokens, head_dim, generator=gen)
        k[:, :, at] = base[:, :, 0, 0] * (nats + 1.5) / head_dim ** 0.5
        v[:, :, at] *= 0.01 if nats < 10 else 0.001
    elif kind == "outlier1e3":
        k[..., 7] *= 1e3
        q[..., 7] *= 1e-4
    elif kind == "outlier1e4":
        k[..., 7] = k[..., 7].clamp(-3, 3) * 1e4
        q[..., 7] *= 1e-5
    else:
        v *= torch.exp(2 * torch.randn(1, 1, tokens, 1, generator=gen).clamp(-1.5, 1.5))
    return [t.to(torch.bfloat16) for t in (k, v, q)]


@pytest.mark.parametrize("kind", ["sink8", "sink12", "sink8late", "outlier1e3", "outlier1e4", "spread"])
@pytest.mark.parametrize("bits,D,gqa,B,KVH,S", [(1, 128, 4, 2, 2, 1500), (2, 128, 4, 40, 4, 700), (2, 64, 2, 2, 2, 900), (3, 128, 4, 2, 2, 1500), (3, 128, 4, 20, 8, 500),
                                                (4, 128, 4, 2, 2, 1500), (4, 128, 8, 2, 2, 1500), (4, 64, 1, 2, 2, 1500)])
def test_error_where_large_factors_do_not_meet(oracle, bits, D, gqa, B, KVH, S, kind):
    """tcgen05 kernel: its fixed-point operands are scaled by the largest products of a step, so that rows as models have them (attention sinks,
    outlier channels) keep the error of an fp32 evaluation, or with two planes that of their values (test_tcgen05_kernel).  Two planes:
    2 bits, head_dim 128, more pairs than SMs."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = unlike_tokens(oracle, kind, B, KVH, S, D, gqa, bits + 10)
    ref = oracle.OracleCacheLayer(bits=bits, group=64, residual=128, alpha_key=2.0, alpha_value=4.0)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, alpha_key=2.0, alpha_value=4.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    with kernel(4):
        got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32)
    assert relative_error(got, attention64(oracle, ref, q, D ** -0.5)) <= (1.2e-4 if bits == 2 and D == 128 else FP32_ERROR)


@pytest.mark.parametrize("bits,D,gqa", [(1, 128, 4), (2, 128, 2), (2, 128, 8), (3, 128, 4), (4, 128, 4), (4, 64, 8), (2, 64, 1)])
def test_nan_stays_nan(oracle, bits, D, gqa):
    """tcgen05 kernel: a NaN in the mask or in a query and an infinite key range make the heads that meet them NaN, as a floating-point
    evaluation does, and no others (integer products have no NaN of their own)."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention, decode_attention_partial
    k, v, q = oracle.synth_kv(3, 2, 500, D, 2 * gqa, seed=bits)
    q[1, gqa, 0, 3] = float("nan")
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    layer._key_scale[2, 0, 1, 5] = float("inf")
    mask = torch.zeros(3, 1, 1, 500)
    mask[0, ..., 70] = float("nan")
    hit = torch.zeros(3, 1, 2 * gqa, D, dtype=torch.bool)
    hit[0], hit[1, :, gqa], hit[2, :, :gqa] = True, True, True
    with kernel(4):
        got = decode_attention(layer, q.cuda(), D ** -0.5, mask.cuda(), out_dtype=torch.float32).cpu()
        acc = decode_attention_partial(layer, q.cuda(), D ** -0.5, mask.cuda())[2].cpu().reshape(got.shape)
    for out in (got, acc):
        assert torch.equal(torch.isnan(out), hit) and bool(torch.isfinite(out[~hit]).all())


@pytest.mark.parametrize("meta", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,D,gqa,B,S", [(1, 128, 4, 3, 128 + 64), (1, 128, 2, 2, 128 + 5 * 64 + 63), (2, 128, 4, 3, 128 + 128), (2, 128, 1, 2, 128 + 3 * 64 + 1), (2, 128, 4, 24, 1111),
                                          (3, 128, 4, 3, 128 + 64 + 17), (3, 128, 1, 2, 128 + 128 + 1), (3, 128, 4, 20, 128 + 9 * 64), (1, 128, 4, 40, 700), (3, 128, 2, 2, 5000),
                                          (4, 128, 4, 3, 128 + 64 + 5), (4, 128, 1, 3, 2500), (4, 128, 8, 3, 700), (4, 128, 8, 20, 1000), (1, 128, 8, 2, 900), (2, 128, 8, 12, 777), (3, 128, 8, 3, 200), (1, 64, 4, 3, 330), (2, 64, 4, 3, 128 + 64 + 9), (2, 64, 2, 24, 600),
                                            (3, 64, 1, 2, 1500), (4, 64, 4, 3, 700), (4, 64, 8, 2, 128 + 128), (3, 64, 4, 20, 900),
                                          # too many pairs or tiles for cluster mode, which takes calls below three tiles per SM
                                          (1, 128, 4, 20, 128 + 64), (2, 128, 4, 20, 128 + 128), (3, 128, 4, 20, 128 + 64 + 17), (1, 128, 2, 2, 128 + 112 * 64 + 63)])
def test_tcgen05_kernel(oracle, bits, D, gqa, B, S, meta):
    """One group, whole and half steps, one tile and many in the residual window, a worker's range over several pairs, ranges that do not
    straddle zero, symmetric ones, masked tokens and sequences.  Two-plane calls round a value to 2^-15 of its side:
    2^-16 / sqrt(3) over a value of 0.4 sides, times a logit of about 3, once for keys and once for values: 6e-5, bounded by twice that."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(B, 8 if B > 3 else 2, S, D, (8 if B > 3 else 2) * gqa, seed=bits * 100 + S)
    k[:, :, :, :3] += 4.0
    v[0] -= 3.0
    k[0, 0, 0::2, 5], k[0, 0, 1::2, 5] = 1.5, -1.5
    ref = oracle.OracleCacheLayer(bits=bits, group=64, residual=128, meta_dtype=meta, alpha_key=2.0, alpha_value=4.0)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, amax_dtype=str(meta)[6:], alpha_key=2.0, alpha_value=4.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    mask = torch.zeros(B, 1, 1, S)
    mask[B // 2, ..., : S - 130] = torch.finfo(torch.bfloat16).min
    bound = 1.2e-4 if bits in (2, 4) and D == 128 and B > 3 and gqa <= 4 else FP32_ERROR
    for m in (None, mask):
        want = attention64(oracle, ref, q, D ** -0.5, m)
        got = decode_attention(layer, q.cuda(), D ** -0.5, None if m is None else m.cuda(), out_dtype=torch.float32)
        assert bool(torch.isfinite(got).all()) and relative_error(got, want) <= bound
    if B > 3:
        return
    for i in range(66):          # the kernel stores the newest token itself; one step flushes
        kn, vn, qn = oracle.synth_kv(B, 2, 1, D, 2 * gqa, seed=9000 + i)
        ref.append(kn, vn)
        got = layer.decode_step(kn.cuda(), vn.cuda(), qn.cuda(), D ** -0.5)
    assert torch.equal(layer.keys.cpu(), ref.keys) and torch.equal(layer.values.cpu(), ref.values)
    assert relative_error(got.float(), attention64(oracle, ref, qn, D ** -0.5)) <= 2.0 ** -8      # bf16 output


@pytest.mark.parametrize("bits,bound", [(2, 1.2e-4), (4, 5e-5)])
def test_error_of_the_unrolled_kernel(oracle, bits, bound):
    """Head_dim 128, group 64, up to four heads, more pairs than SMs: the unrolled kernel's table keeps 11 bits and a nominal
    remainder.  The remainder's ratio is off by up to the width of a zero code's bin, so an entry is wrong by up to
    2^-12 (half an fp16 ulp) at 2 bits, a fourth of that at 4 bits; sums over channels and tokens average it down by half."""
    import muzero_b200 as mz
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(20, 8, 400, 128, 32, seed=bits)
    ref = oracle.OracleCacheLayer(bits=bits, group=64, residual=128, alpha_key=2.0, alpha_value=2.0)
    ref.append(k, v)
    layer = mz.MuZeroCacheLayer(mz.MuZeroConfig(bits=bits, alpha_key=2.0, alpha_value=2.0))
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    got = decode_attention(layer, q.cuda(), 128 ** -0.5, out_dtype=torch.float32)
    assert relative_error(got, attention64(oracle, ref, q, 128 ** -0.5)) <= bound


@pytest.mark.parametrize("which", [0, 4])
@pytest.mark.parametrize("bits,D,gqa,B,S,residual", [(4, 128, 8, 2, 1200, 128), (2, 128, 4, 2, 1200, 256), (3, 64, 1, 3, 700, 256), (4, 128, 8, 20, 400, 128)])
def test_workspace_bound_covers_every_split_count(oracle, bits, D, gqa, B, S, residual, which):
    """The bound that holds for any token count also holds for two plans of as many workers as explicit splits ask for."""
    import ctypes
    import muzero_b200 as mz
    from muzero_b200.cache.attention import build_decode_args
    from muzero_b200.kernels._cabi import load_library
    k, v, q = oracle.synth_kv(B, 4, S, D, 4 * gqa, seed=bits)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=residual, alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    lib = load_library()
    with kernel(which):
        a = build_decode_args(layer, q.cuda(), D ** -0.5, None, None)
        for a.splits in range(0, 40):
            need, bound = lib.mz_decode_workspace_bytes(ctypes.byref(a)), lib.mz_decode_workspace_bound(ctypes.byref(a))
            assert 0 < need <= bound, (a.splits, need, bound)


def planned_kernel(layer, q, splits=0):
    """mz_debug_decode_kernel of a call: 2 general kernel in clusters, 4 unrolled kernel, 4 + n tcgen05 kernel with n bytes per value."""
    import ctypes
    from muzero_b200.cache.attention import build_decode_args
    from muzero_b200.kernels._cabi import load_library
    return load_library().mz_debug_decode_kernel(ctypes.byref(build_decode_args(layer, q, 1.0, None, None, splits=splits)))


def caches(oracle, k, v, bits, **kw):
    """The same keys and values in the oracle's cache and on the GPU, group 64 and a residual window of 128."""
    import muzero_b200 as mz
    meta = kw.pop("meta", torch.float16)
    ref = oracle.OracleCacheLayer(bits=bits, group=64, residual=128, meta_dtype=meta, **kw)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, amax_dtype=str(meta)[6:], **kw)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {"materialize_full_kv": False})
    return ref, layer


# two planes: see test_tcgen05_kernel
TWO_PLANE_ERROR = 1.2e-4


@pytest.mark.parametrize("meta", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits,D,gqa,B,S", [(1, 128, 1, 2, 128 + 64), (1, 128, 8, 3, 700), (1, 64, 2, 2, 128 + 128), (2, 128, 4, 3, 128 + 64 + 63), (2, 128, 1, 2, 900), (2, 128, 8, 2, 330),
                                            (2, 64, 4, 3, 1111), (2, 64, 8, 2, 200), (3, 128, 1, 2, 128 + 128 + 1), (3, 128, 2, 3, 777), (3, 128, 8, 2, 600), (3, 64, 8, 3, 300),
                                            (4, 128, 1, 3, 128 + 64 + 5), (4, 128, 2, 2, 500), (4, 128, 4, 3, 2500), (4, 128, 8, 3, 1000), (4, 64, 1, 2, 330), (4, 64, 8, 3, 640)])
def test_tcgen05_kernel_takes_the_new_token(oracle, bits, D, gqa, B, S, meta):
    """Every width, head set and head_dim on the tcgen05 kernel itself, whatever the automatic choice: decode steps whose new token the kernel
    stores (eight heads: two workers read it and one stores it), across a flush."""
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(B, 2, S, D, 2 * gqa, seed=bits * 100 + S)
    k[:, :, :, :3] += 4.0
    v[0] -= 3.0
    ref, layer = caches(oracle, k, v, bits, alpha_key=2.0, alpha_value=4.0, meta=meta)
    two = bits == 2 and D == 128
    bound = TWO_PLANE_ERROR if two else FP32_ERROR
    with kernel(4):
        assert planned_kernel(layer, q.cuda()) == 4 + (1 if bits == 1 else 2 if two else 3)
        for i in range(66):
            kn, vn, qn = oracle.synth_kv(B, 2, 1, D, 2 * gqa, seed=9000 + i)
            ref.append(kn, vn)
            got = layer.decode_step(kn.cuda(), vn.cuda(), qn.cuda(), D ** -0.5)
            if i in (0, 65):
                want = attention64(oracle, ref, qn, D ** -0.5)
                assert relative_error(got.float(), want) <= 2.0 ** -8      # bf16 output
                assert relative_error(decode_attention(layer, qn.cuda(), D ** -0.5, out_dtype=torch.float32), want) <= bound
    assert torch.equal(layer.keys.cpu(), ref.keys) and torch.equal(layer.values.cpu(), ref.values)


@pytest.mark.parametrize("vs,ks,qs,meta", [(1e-4, 1.0, 1.0, torch.float16), (1e-6, 1.0, 1.0, torch.float32), (1e5, 1.0, 1.0, torch.float32),
                                           (1e5, 1.0, 1.0, torch.bfloat16), (1.0, 1e-4, 1e4, torch.float16), (1.0, 1e5, 1e-5, torch.float32)])
@pytest.mark.parametrize("bits,D,gqa", [(1, 128, 2), (2, 64, 4), (3, 128, 4), (4, 128, 8), (4, 64, 1)])
def test_tcgen05_error_at_any_scale(oracle, bits, D, gqa, vs, ks, qs, meta):
    """test_error_at_any_scale on the tcgen05 kernel."""
    from muzero_b200.cache.attention import decode_attention
    k, v, q = (t.float() for t in oracle.synth_kv(2, 2, 700, D, 2 * gqa, seed=bits))
    v[..., :32] *= 1e-3
    k, v, q = ((t * f).to(torch.bfloat16) for t, f in ((k, ks), (v, vs), (q, qs)))
    ref, layer = caches(oracle, k, v, bits, alpha_key=2.0, alpha_value=2.0, meta=meta)
    want = attention64(oracle, ref, q, D ** -0.5)
    with kernel(4):
        got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32)
    assert bool(torch.isfinite(got).all())
    for part in (slice(0, 32), slice(32, D)):
        assert relative_error(got[..., part], want[..., part]) <= (FP32_ERROR if part.start else SHARED_GROUP_ERROR)


@pytest.mark.parametrize("bits,D,gqa", [(1, 128, 4), (2, 128, 2), (3, 128, 4), (4, 64, 8), (4, 128, 8)])
def test_tcgen05_infinite_range_stays_in_its_group(oracle, bits, D, gqa):
    """test_an_infinite_range_stays_in_its_group on the tcgen05 kernel."""
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(2, 2, 500, D, 2 * gqa, seed=bits)
    ref, layer = caches(oracle, k, v, bits, alpha_key=2.0, alpha_value=2.0)
    want = attention64(oracle, ref, q, D ** -0.5)
    last = D // 64 - 1
    layer._value_scale[0, 1, 5, last] = float("inf")
    with kernel(4):
        got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32).cpu()
    hit = torch.zeros(got.shape, dtype=torch.bool)
    hit[0, :, gqa:, 64 * last:64 * last + 64] = True
    assert not bool(torch.isfinite(got[hit]).any())
    assert relative_error(got[~hit], want[~hit]) <= (TWO_PLANE_ERROR if bits == 2 else FP32_ERROR)


@pytest.mark.parametrize("B,KVH,S,planned", [(1, 8, 3900, 7), (3, 2, 4992, 7), (3, 2, 4928, 6), (3, 2, 4864, 6), (20, 8, 400, 6), (1, 8, 1500, 2)])
def test_bytes_per_value_at_2_bits(oracle, B, KVH, S, planned):
    """Calls that cluster mode would serve keep the error of its fp32 evaluation on the tcgen05 kernel too (three planes); those that the unrolled
    kernel would serve take two planes, whose error is below that kernel's.  On both sides of the line; the call's own choice."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line is drawn per SM")
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(B, KVH, S, 128, 4 * KVH, seed=S)
    ref, layer = caches(oracle, k, v, 2, alpha_key=2.0, alpha_value=2.0)
    assert planned_kernel(layer, q.cuda()) == planned
    got = decode_attention(layer, q.cuda(), 128 ** -0.5, out_dtype=torch.float32)
    assert relative_error(got, attention64(oracle, ref, q, 128 ** -0.5)) <= (TWO_PLANE_ERROR if planned == 6 else FP32_ERROR)


@pytest.mark.parametrize("gqa", [1, 2, 4])
def test_unrolled_kernel_at_2_bits_with_splits(oracle, gqa):
    """Explicit splits are what the unrolled kernel's 2-bit instances serve; the bound is that of test_error_of_the_unrolled_kernel."""
    from muzero_b200.cache.attention import decode_attention
    k, v, q = oracle.synth_kv(20, 8, 400, 128, 8 * gqa, seed=2)
    ref, layer = caches(oracle, k, v, 2, alpha_key=2.0, alpha_value=2.0)
    want = attention64(oracle, ref, q, 128 ** -0.5)
    for splits in (1, 3):
        assert planned_kernel(layer, q.cuda(), splits) == 4
        got = decode_attention(layer, q.cuda(), 128 ** -0.5, out_dtype=torch.float32, splits=splits)
        assert relative_error(got, want) <= 1.2e-4


@pytest.mark.parametrize("bits,gqa,B,KVH,S,planned", [(4, 4, 33, 8, 592, 3), (4, 4, 21, 8, 946, 3), (2, 4, 29, 4, 733, 2), (4, 8, 2, 8, 16198, 3), (4, 4, 40, 4, 3000, 3), (4, 2, 1, 4, 34849, 7)])
def test_residual_tiles_weigh_in_the_choice_at_head_dim_64(oracle, bits, gqa, B, KVH, S, planned):
    """Calls with about as many residual as packed tiles stay with the general kernel (20 to 45 % faster there), a long one goes to the tcgen05
    kernel (twice as fast there)."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line is drawn per SM")
    import muzero_b200 as mz
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, alpha_key=2.0, alpha_value=2.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    k = torch.randn(B, KVH, S, 64, device="cuda", dtype=torch.bfloat16)
    layer.update(k, k.clone(), {"materialize_full_kv": False})
    assert planned_kernel(layer, k.new_zeros(B, KVH * gqa, 1, 64)) == planned
