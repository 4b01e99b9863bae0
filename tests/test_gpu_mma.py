"""GPU: the tensor-core decode kernel at the edges of its tiles, widths and head sets, in its cluster and flat forms."""
import pytest
import torch

from test_gpu_attention import SPLIT_TOL, check_output

pytestmark = pytest.mark.gpu


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
