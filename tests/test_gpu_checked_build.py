"""GPU: the checked build of the library (compiled with -DMZ_BOUNDS).

Guarded global stores compare their index with the extent the host passed; an access outside it is skipped
and counted, never trapped, so the CUDA context stays usable.  The checked library is a second shared
object, selected through MUZERO_B200_LIB, so it is exercised in a child process: small shapes through the
cache layer (prefill flush, decode steps with every decode-attention kernel, a batch gather) must leave the
violation count at zero and still agree with the CPU oracle; a flush into a store that is declared full must
be counted and must leave the store untouched.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKED_LIB = os.path.join(ROOT, "muzero_b200", "lib", "libmuzero_b200_bounds.so")

CHILD = r"""
import ctypes, sys, torch
sys.path.insert(0, {root!r}); sys.path.insert(0, {root!r} + "/tests")
from conftest import load_oracle
import muzero_b200 as mz
from muzero_b200.cache.attention import decode_attention
from muzero_b200.kernels._cabi import check, load_library, stream_ptr
lib = load_library()
orc = load_oracle()

def violations(reset=0):
    i, n, site = ctypes.c_longlong(), ctypes.c_longlong(), ctypes.c_int()
    c = lib.mz_bounds_violations(ctypes.byref(i), ctypes.byref(n), ctypes.byref(site), reset)
    return c, i.value, n.value, site.value

assert violations()[0] == 0, "not a checked build, or a dirty record: %r" % (violations(),)
for bits, gqa in ((4, 4), (2, 2), (3, 1)):
    KVH = 2
    k, v, q = orc.synth_kv(3, KVH, 64 * 7 + 50, 128, KVH * gqa, seed=900 + bits)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {{"materialize_full_kv": False}})
    ref = orc.OracleCacheLayer(bits=bits, group=64, residual=128)
    ref.append(k, v)
    want = orc.decode_attention_oracle(q, ref, 0.088, gqa, compute_dtype=torch.float32)
    for which in (1, 2, 3, 4):                      # generic, SIMT tiles, mma.sync, tcgen05 (where they apply)
        prev = lib.mz_debug_force_kernel(which)
        try:
            got = decode_attention(layer, q.cuda(), 0.088, out_dtype=torch.float32)
        finally:
            lib.mz_debug_force_kernel(prev)
        err = (got.cpu() - want).abs().max().item()
        assert err <= 2e-3, (bits, gqa, which, err)
    # decode steps across a flush, then a batch gather
    for step in range(70):
        kn, vn, _ = orc.synth_kv(3, KVH, 1, 128, KVH * gqa, seed=5000 + step)
        if step % 2:
            layer.update(kn.cuda(), vn.cuda(), {{"materialize_full_kv": False}})
        else:                                       # the decode kernel stores the new token itself
            layer.decode_step(kn.cuda(), vn.cuda(), q.cuda(), 0.088)
    layer._full_kv()
    mz.roundtrip(k[:, :, :448].cuda(), v[:, :, :448].cuda(), bits=bits, q_group_size=64)
    layer.batch_select_indices(torch.tensor([2, 0], device="cuda"))
    c = violations()
    assert c[0] == 0, (bits, c)

# a store declared full: the flush must skip every store, count them, and change nothing
k, v, q = orc.synth_kv(2, 2, 64 * 4 + 128, 128, 8, seed=77)
layer = mz.MuZeroCacheLayer(mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128))
layer.update(k.cuda(), v.cuda(), {{"materialize_full_kv": False}})
assert layer.keys.shape[2] >= 64
s = layer._store_struct()
bufs = layer._bufs
before = {{n: t.clone() for n, t in bufs.items()}}
s.k_groups = bufs["pk"].shape[2]                   # no room left in either store
s.v_tokens = bufs["pv"].shape[2]
check(lib.mz_flush_kv(ctypes.byref(s), 64, 1e-8, stream_ptr(torch.device("cuda"))), "mz_flush_kv")
count, index, extent, site = violations(reset=1)
assert count > 0 and index >= extent and 1 <= site <= 6, (count, index, extent, site)
for n, t in bufs.items():                         # bit patterns: unused capacity is uninitialised and may hold NaN
    assert torch.equal(t.view(torch.uint8), before[n].view(torch.uint8)), n
assert violations()[0] == 0                        # cleared

# a flush that moves what stays dense into a window declared four rows too short (its memory is not): the rows outside are
# skipped and counted, those inside arrive
s = layer._store_struct()
layer._ensure_store(s.k_groups + 1, s.v_tokens + 64)
s = layer._store_struct()
stay, cols = s.res_len - 64, 128
win = [torch.zeros(2, 2, stay, cols, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
short = (stay - 4) * cols
check(lib.mz_flush_kv_move(ctypes.byref(s), 64, 0, 64, win[0].data_ptr(), win[1].data_ptr(), 2 * stay * cols, short, cols, 1e-8,
                           stream_ptr(torch.device("cuda"))), "mz_flush_kv_move")
moved = violations(reset=1)
assert moved[0] == 2 * 2 * 4 * cols // 8 and moved[3] == 23, moved
got = win[0].reshape(2, -1)[:, : 2 * short].reshape(2, 2, stay - 4, cols)
assert torch.equal(got, layer.keys[:, :, 64:64 + stay - 4])
torch.cuda.synchronize()
print("CHECKED-BUILD-OK", count, site)
"""


def test_checked_build_small_shapes():
    if not os.path.exists(CHECKED_LIB):
        pytest.skip("checked library not built (python -m muzero_b200.build --bounds)")
    env = dict(os.environ, MUZERO_B200_LIB=CHECKED_LIB)
    res = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=900)
    assert res.returncode == 0 and "CHECKED-BUILD-OK" in res.stdout, res.stdout[-2000:] + res.stderr[-4000:]


WAITS_CHILD = r"""
import sys, torch
sys.path.insert(0, {root!r}); sys.path.insert(0, {root!r} + "/tests")
from conftest import load_oracle
import muzero_b200 as mz
from muzero_b200.cache.attention import decode_attention
from muzero_b200.kernels._cabi import load_library
lib, orc = load_library(), load_oracle()
lib.mz_debug_force_kernel(4)
for bits, D, gqa, B, S in ((1, 128, 4, 2, 500), (2, 128, 2, 20, 500), (3, 64, 1, 2, 500), (4, 128, 8, 2, 500), (3, 128, 4, 20, 1000)):
    k, v, q = orc.synth_kv(B, 8, S, D, 8 * gqa, seed=bits)
    ref = orc.OracleCacheLayer(bits=bits, group=64, residual=128, alpha_key=2.0, alpha_value=4.0)
    ref.append(k, v)
    cfg = mz.MuZeroConfig(bits=4, q_group_size=64, residual_length=128, alpha_key=2.0, alpha_value=4.0)
    cfg.bits = bits
    layer = mz.MuZeroCacheLayer(cfg)
    layer.update(k.cuda(), v.cuda(), {{"materialize_full_kv": False}})
    assert lib.mz_debug_fail_waits(1) == 0
    got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32).cpu()
    assert lib.mz_debug_fail_waits(0) == 1
    assert bool(torch.isnan(got).all()), (bits, D, gqa)
    got = decode_attention(layer, q.cuda(), D ** -0.5, out_dtype=torch.float32).cpu()
    want = orc.decode_attention_oracle(q, ref, D ** -0.5, gqa, compute_dtype=torch.float32)
    assert (got - want).abs().max().item() <= 2e-3, (bits, D, gqa)
    # and its stores of the newest token, across a flush
    for step in range(66):
        kn, vn, qn = orc.synth_kv(B, 8, 1, D, 8 * gqa, seed=5000 + step)
        layer.decode_step(kn.cuda(), vn.cuda(), qn.cuda(), D ** -0.5)
    assert torch.equal(layer.keys[:, :, -1:].cpu(), kn) and torch.equal(layer.values[:, :, -1:].cpu(), vn)
assert lib.mz_bounds_violations(None, None, None, 0) == 0
print("WAITS-OK")
"""


def test_a_wait_that_runs_out_gives_nan():
    """tcgen05 kernel, every wait run out at once: every worker gives up, and the output says so; the next call is right again."""
    if not os.path.exists(CHECKED_LIB):
        pytest.skip("checked library not built (python -m muzero_b200.build --bounds)")
    env = dict(os.environ, MUZERO_B200_LIB=CHECKED_LIB)
    res = subprocess.run([sys.executable, "-c", WAITS_CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and "WAITS-OK" in res.stdout, res.stdout[-2000:] + res.stderr[-4000:]
