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
    out, lse = rt.gqa_decode(dq, dk, dv, kv_lens=util.to_cuda(lens))
    f32, _ = rt.gqa_decode(dq, dk, dv, kv_lens=util.to_cuda(lens), out_dtype=torch.float32)
    rec = rt.gqa_decode_record(dq, dk, dv, kv_lens=util.to_cuda(lens))
    torch.cuda.synchronize()
    util.check_output(util.to_np(out), ref)
    util.check_lse(util.to_np(lse), ref_lse)
    assert torch.equal(f32.to(torch.bfloat16), out)
    assert torch.equal(rec[:, :D], f32.reshape(-1, D)) and torch.equal(rec[:, D], lse.reshape(-1))
    # one sequence, the length known to the host
    out1, lse1 = rt.gqa_decode(dq[-1:], dk[-1:], dv[-1:], kv_len=int(lens[-1]))
    util.check_output(util.to_np(out1), ref[-1:])
    util.check_lse(util.to_np(lse1), ref_lse[-1:])


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


@pytest.mark.skipif("RT_ATTN_DECODE_CLUSTER" in os.environ, reason="the child process itself")
@pytest.mark.parametrize("size", ["2", "4", "8", "16"])
def test_every_cluster_size(size):
    run_tests_with("RT_ATTN_DECODE_CLUSTER", size, "test_gpu_decode_cluster.py", "cluster_parts")


@pytest.mark.skipif("RT_ATTN_DECODE_CLUSTER" in os.environ, reason="the child process itself")
def test_other_splits_without_clusters():
    run_tests_with("RT_ATTN_DECODE_CLUSTER", "0", "test_gpu_dispatch_edges.py", "decode_splits")
    run_tests_with("RT_ATTN_DECODE_CLUSTER", "0", "test_gpu_decode.py")
