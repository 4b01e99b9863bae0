"""GPU: the packed quantizer, the dense read-back, the fp32 quantizer and the alpha statistics against the oracle."""
import numpy as np
import pytest
import torch

from conftest import bits16

pytestmark = pytest.mark.gpu


def _block(oracle, B, KVH, S, D, dtype, seed):
    """K / V with rows at the edges of the quantizer: constant, one-sided (anchor 0 and 1), tiny."""
    k, v, _ = oracle.synth_kv(B, KVH, S, D, KVH, seed=seed)
    k, v = k.float().clamp(-6e4, 6e4), v.float()
    k[0, 0, :, 0], k[0, 0, :, 1], k[0, 0, :, 2] = 1.5, k[0, 0, :, 1].abs() + 0.1, -k[0, 0, :, 2].abs() - 0.1
    k[0, 0, :, 3] *= 1e-4
    v[0, 0, 1], v[0, 0, 2], v[0, 0, 3] = -2.0, v[0, 0, 2].abs() + 0.1, -v[0, 0, 3].abs() - 0.1
    if dtype == torch.float16:       # a zero range is NaN in the reference at fp16
        k[0, 0, :, 0] += torch.arange(S) % 2
        v[0, 0, 1] += torch.arange(D) % 2
    return k.to(dtype), v.to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,group", [(64, 32), (64, 64), (128, 32), (128, 64), (128, 128)])
@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 7, 8])
def test_flush_and_read_back(oracle, bits, D, group, dtype):
    import muzero_b200 as mz
    S = 128 + 3 * group + 5
    k, v = _block(oracle, 1, 3, S, D, dtype, seed=bits + group)
    ref = oracle.OracleCacheLayer(bits=bits, group=group, residual=128)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=group, residual_length=128)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda().transpose(1, 2).contiguous().transpose(1, 2), v.cuda().transpose(1, 2).contiguous().transpose(1, 2),
                 {"materialize_full_kv": False})
    assert [layer._selected_alpha_key, layer._selected_alpha_value] == [ref.alpha_key, ref.alpha_value]
    for mine, theirs in ((layer._key_mn, ref.k_mn), (layer._key_scale, ref.k_scale), (layer._value_mn, ref.v_mn),
                         (layer._value_scale, ref.v_scale)):
        assert np.array_equal(bits16(mine), bits16(theirs))
    assert torch.equal(layer._packed_key_q.cpu(), ref.packed_k)
    assert torch.equal(layer._packed_value_q.cpu(), ref.packed_v)
    full_k, full_v = layer._full_kv()
    assert np.array_equal(bits16(full_k), bits16(torch.cat([ref.key_prefix(dtype), ref.keys], dim=2)))
    assert np.array_equal(bits16(full_v), bits16(torch.cat([ref.value_prefix(dtype), ref.values], dim=2)))


@pytest.mark.parametrize("alpha", [2.0, 16.0])
@pytest.mark.parametrize("bits,D,group", [(1, 64, 32), (4, 128, 64), (3, 128, 128), (8, 64, 64)])
def test_roundtrip_equals_rows_in_fp32(oracle, bits, D, group, alpha):
    import muzero_b200 as mz
    k, v = _block(oracle, 2, 2, 3 * group, D, torch.bfloat16, seed=bits)
    got = mz.roundtrip(k.cuda(), v.cuda(), bits=bits, q_group_size=group, alpha_key=alpha, alpha_value=alpha)

    def through(rows):
        q = oracle.quantize_rows_oracle(rows.float(), bits, alpha, 1e-8, torch.float16)
        return oracle.dequantize_rows_oracle(*q, bits, alpha, group, torch.bfloat16)
    b, h, s, d = k.shape
    want_k = through(oracle.key_rows(k, group)).reshape(b, h, s // group, d, group).transpose(3, 4).reshape(k.shape)
    want_v = through(oracle.value_rows(v, group)).reshape(v.shape)
    # torch's fp32 log1p is not correctly rounded everywhere: codes may differ where a position falls on a half
    for mine, want in ((got[0], want_k), (got[1], want_v)):
        assert (mine.cpu() != want).float().mean().item() <= 1e-5


@pytest.mark.parametrize("power,shift,group", [(1, 0.0, 64), (3, 0.0, 32), (1, 1.0, 64)])
def test_alpha_statistics(oracle, power, shift, group):
    from muzero_b200.quantizer import device_alphas, select_alpha
    k, _ = _block(oracle, 2, 3, 4 * group, 128, torch.bfloat16, seed=group)
    k = (k.float() ** power + shift).to(torch.bfloat16)
    for bits in (1, 3, 8):
        want = [oracle.select_alpha_oracle(oracle.key_rows(k, group), bits=bits, group=group, kind="key", max_points=5000),
                oracle.select_alpha_oracle(oracle.value_rows(k, group), bits=bits, group=group, kind="value", max_points=5000)]
        assert device_alphas([(k.cuda(), "key", 1), (k.cuda(), "value", 0)], bits=bits, q_group_size=group, max_points=5000) == want
        for kind in ("key", "value"):
            assert select_alpha(k.cuda(), bits=bits, q_group_size=group, kind=kind) == \
                oracle.select_alpha_oracle(k, bits=bits, group=group, kind=kind)
