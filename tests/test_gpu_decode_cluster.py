"""Decode launches in which a cluster of CTAs streams a sequence and merges its parts itself (csrc/decode_tc.cu,
merge_decode_cluster), against the CPU oracle: every cluster size, head dim and group size, and lengths at which CTAs of
a cluster get nothing, a ragged last block, or all of a part.  The size is a launch rule's choice that an override sets, and the
library reads overrides once per process, so each size runs in a child process; so do the other rules of the split,
which clusters take over at these sizes."""
import os

import numpy as np
import pytest

from tests import util
from tests.test_gpu_overrides import run_tests_with

pytestmark = pytest.mark.gpu


def _check_scratch(q, k, v, lens, want):
    """Under an override that sets a cluster's size no chunk partial is written: the launch took clusters."""
    import torch
    import rustorch_b200 as rt
    from rustorch_b200 import _lib
    size = int(os.environ.get("RT_ATTN_DECODE_CLUSTER", "0"))
    if size == 0:
        return
    (B, Hq, D), (Hkv, S) = q.shape, k.shape[1:3]
    ws = torch.full((rt.decode_workspace_bytes(B, Hq, Hkv, D, S),), 0xff, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(want)
    rc = _lib.lib().rt_gqa_decode_bf16(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, None, B, Hq, Hkv, D, S,
                                       lens.data_ptr(), 0, 0, -1, -1.0, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(out, want) and ws.numel() > 0 and bool((ws == 0xff).all())


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("G,Hkv", [(1, 2), (2, 1), (4, 2), (8, 1)])
def test_cluster_parts(oracle, D, G, Hkv):
    """Lengths at the edges of a part of 64 tokens for 1 to 16 parts, an empty sequence, NaN bits beyond each length."""
    import torch
    import rustorch_b200 as rt
    lens = np.array([0, 1, 63, 64, 65, 129, 257, 1000], dtype=np.int32)
    B, S = len(lens), 1100
    q = util.normal_bf16(oracle, (B, Hkv * G, D), 1)
    k, v = (util.normal_bf16(oracle, (B, Hkv, S, D), s) for s in (2, 3))
    _, ref, ref_lse = oracle.gqa_decode_cache(q, k, v, lens)
    dq, dk, dv = (util.to_cuda_bf16(x) for x in (q, k, v))
    for b, n in enumerate(lens):
        dk[b, :, n:] = float("nan")
        dv[b, :, n:] = float("nan")
    # all of them, and pairs: 16 CTAs of D = 256 for each of 16 (sequence, KV head) groups are not resident at once
    for part in [slice(0, B)] + [slice(i, i + 2) for i in range(0, B, 2)]:
        tq, tk, tv, tl = dq[part], dk[part], dv[part], util.to_cuda(lens[part])
        out, lse = rt.gqa_decode(tq, tk, tv, kv_lens=tl)
        f32, _ = rt.gqa_decode(tq, tk, tv, kv_lens=tl, out_dtype=torch.float32)
        rec = rt.gqa_decode_record(tq, tk, tv, kv_lens=tl)
        torch.cuda.synchronize()
        util.check_output(util.to_np(out), ref[part])
        util.check_lse(util.to_np(lse), ref_lse[part])
        assert torch.equal(f32.to(torch.bfloat16), out)
        assert torch.equal(rec[:, :D], f32.reshape(-1, D)) and torch.equal(rec[:, D], lse.reshape(-1))
        if part.stop - part.start == 2:
            _check_scratch(tq, tk, tv, tl, out)
    # one sequence, the length known to the host
    out1, lse1 = rt.gqa_decode(dq[-1:], dk[-1:], dv[-1:], kv_len=int(lens[-1]))
    util.check_output(util.to_np(out1), ref[-1:])
    util.check_lse(util.to_np(lse1), ref_lse[-1:])


def test_lse_of_a_merge():
    """The log-sum-exp that a cluster merges, against 64 bits: a rounding of the result (LSE in 4..8: 4.8e-7 / sqrt(12)) and a
    logarithm within one unit of its last place (at most 4.8e-7 / sqrt(3)) make 3.1e-7 rms.  Measured 2.5e-7; 4.2e-7 with lg2.approx."""
    import torch
    import rustorch_b200 as rt
    B, Hq, Hkv, D, S = 1, 32, 8, 128, 300
    err = []
    for seed in range(24):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q, k, v = (torch.randn(s, device="cuda", generator=g).to(torch.bfloat16) for s in ((B, Hq, D), (B, Hkv, S, D), (B, Hkv, S, D)))
        _, lse = rt.gqa_decode(q, k, v, kv_len=S)
        s = torch.einsum("bhd,bhsd->bhs", q.double(), k.double().repeat_interleave(Hq // Hkv, 1)) / D ** 0.5
        err.append(lse.double() - torch.logsumexp(s, -1))
    assert torch.cat(err).pow(2).mean().sqrt().item() < 3.2e-7


@pytest.mark.parametrize("offset", [1, 2, 3])
@pytest.mark.parametrize("n,D", [(1000, 64), (1000, 128), (1000, 256), (40, 128)])
def test_output_of_any_element_alignment(n, D, offset):
    """An output that starts 1, 2 or 3 elements into a buffer gets the bits of an aligned one: lengths that clusters take,
    and one that a single CTA does."""
    import torch
    import rustorch_b200 as rt
    g = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (torch.randn(s, dtype=torch.bfloat16, device="cuda", generator=g) for s in ((2, 8, D), (2, 2, n, D), (2, 2, n, D)))
    want, _ = rt.gqa_decode(q, k, v, kv_len=n)
    buf = torch.full((q.numel() + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    out, _ = rt.gqa_decode(q, k, v, kv_len=n, out=buf[offset:offset + q.numel()].view(q.shape))
    torch.cuda.synchronize()
    assert out.data_ptr() % 8 == 2 * offset and torch.equal(out, want)
    assert bool((buf[:offset] == 7.0).all()) and bool((buf[offset + q.numel():] == 7.0).all())


def test_pushed_record_of_any_alignment():
    """rt_gqa_decode_record_push_bf16 with a record that is no slot and lies 4 to 12 bytes off a 16-byte boundary: taken at a
    length that clusters serve for an aligned one, delivered to every peer, and equal up to the roundings of P."""
    import ctypes
    import torch
    import rustorch_b200 as rt
    from rustorch_b200 import _lib
    B, Hq, Hkv, D, S, world = 1, 8, 2, 128, 1000, 2
    rows = B * Hq
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(s, dtype=torch.bfloat16, device="cuda", generator=g) for s in ((B, Hq, D), (B, Hkv, S, D), (B, Hkv, S, D)))
    want = rt.gqa_decode_record(q, k, v, kv_len=S)
    ws = torch.empty(rt.decode_workspace_bytes(B, Hq, Hkv, D, S), dtype=torch.uint8, device="cuda")
    buf = torch.empty(rows * (D + 1) + 4, dtype=torch.float32, device="cuda")
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    for off in range(4):
        slots = [torch.full((rows, D + 1), float("nan"), device="cuda") for _ in range(world)]
        flags = torch.zeros(world, dtype=torch.int32, device="cuda")
        p_slots = (ctypes.c_void_p * world)(*[t.data_ptr() for t in slots])
        p_flags = (ctypes.c_void_p * world)(*[flags.data_ptr() + 4 * r for r in range(world)])
        rc = _lib.lib().rt_gqa_decode_record_push_bf16(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), buf.data_ptr() + 4 * off, p_slots, p_flags, world, 5, done.data_ptr(), B, Hq, Hkv,
            D, S, None, S, 0, -1, -1.0, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        rec = buf[off:off + rows * (D + 1)].view(rows, D + 1)
        # another cut rounds P to bf16 against other running maxima: 2^-9 a weight, 2^-9 / sqrt(keys) an element, times 16
        assert (rec - want).abs().max().item() < 1e-3
        assert all(torch.equal(t, rec) for t in slots) and flags.tolist() == [5] * world and int(done.item()) == 0


@pytest.mark.skipif("RT_ATTN_DECODE_CLUSTER" in os.environ, reason="the child process itself")
@pytest.mark.parametrize("size", ["2", "4", "8", "16"])
def test_every_cluster_size(size):
    run_tests_with("RT_ATTN_DECODE_CLUSTER", size, "test_gpu_decode_cluster.py", "cluster_parts")


@pytest.mark.skipif("RT_ATTN_DECODE_CLUSTER" in os.environ, reason="the child process itself")
def test_other_splits_without_clusters():
    run_tests_with("RT_ATTN_DECODE_CLUSTER", "0", "test_gpu_dispatch_edges.py", "decode_splits")
    run_tests_with("RT_ATTN_DECODE_CLUSTER", "0", "test_gpu_decode.py")
