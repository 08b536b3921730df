"""The f32 forward where a cluster of CTAs shares the keys of a row block (csrc/prefill_simt.cu, kSplit): launches of few row blocks,
keys at the edges of a CTA's share of 64-key tiles, against the CPU oracle at the f32 kernels' 1e-4.  The size is a launch
rule's choice that an override sets for every launch, and the library reads overrides once per process: each size, and the launch
without clusters, runs in a child process."""
import os

import numpy as np
import pytest

from tests import util
from tests.test_gpu_overrides import run_tests_with

pytestmark = pytest.mark.gpu


def _check(out, lse, ref, ref_lse):
    out, lse = util.to_np(out), util.to_np(lse)
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    assert np.nanmax(np.abs(out - ref), initial=0.0) < 1e-4
    fine = np.isfinite(ref_lse)
    assert np.array_equal(fine, np.isfinite(lse)) and np.abs(lse[fine] - ref_lse[fine]).max(initial=0.0) < 1e-4


@pytest.mark.parametrize("D", [7, 64, 80, 128])
@pytest.mark.parametrize("N", [129, 256, 257, 511, 513, 1100])
@pytest.mark.parametrize("causal", [False, True])
def test_shared_row_blocks(oracle, N, D, causal):
    import rustorch_b200 as rt
    q, k, v = (oracle.fill_normal((1, 2, N, D), s) for s in (1, 2, 3))
    out, lse = rt.prefill_f32(*(util.to_cuda(x) for x in (q, k, v)), causal=causal)
    _, ref, ref_lse = oracle.flash_forward_ext(q, k, v, causal=causal)
    _check(out, lse, ref, ref_lse)


def test_shares_without_a_visible_key(oracle):
    """Keep flags that hide whole tiles, all keys of a sequence (NaN rows), or all but one."""
    import rustorch_b200 as rt
    N = 640
    q, k, v = (oracle.fill_normal((4, 1, N, 64), s) for s in (4, 5, 6))
    keep = np.zeros((4, N), dtype=np.uint8)
    keep[0, 500:510] = 1
    keep[2, 63] = 1
    keep[3, :] = 1
    out, lse = rt.prefill_f32(*(util.to_cuda(x) for x in (q, k, v)), key_keep=util.to_cuda(keep))
    _, ref, ref_lse = oracle.flash_forward_ext(q, k, v, keep=keep)
    _check(out, lse, ref, ref_lse)


@pytest.mark.parametrize("Nq,Nkv,Hq,Hkv,D", [(64, 4096, 2, 1, 128), (100, 2048, 4, 2, 64), (130, 700, 4, 1, 80)])
@pytest.mark.parametrize("causal", [False, True])
def test_few_rows_against_many_keys(Nq, Nkv, Hq, Hkv, D, causal):
    """Grouped heads, lengths down to less than the first CTA's first tile (and none), offsets of the rows under a causal mask, at
    shapes where the rule itself takes large clusters.  Against attention in 64 bits."""
    import torch
    import rustorch_b200 as rt
    lens = [0, 1, 65, 129, Nkv // 2 + 3, Nkv]
    B = len(lens)
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k, v = (torch.randn(s, device="cuda", generator=g) for s in ((B, Hq, Nq, D), (B, Hkv, Nkv, D), (B, Hkv, Nkv, D)))
    kv_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    offs = torch.tensor([max(0, n - Nq) for n in lens], dtype=torch.int32, device="cuda")
    pos = torch.arange(Nkv, device="cuda")
    for rows in (slice(0, B), slice(B - 1, B)):  # (a launch of few row blocks too)
        n, o = kv_lens[rows], offs[rows]
        out, lse = rt.prefill_f32(q[rows], k[rows], v[rows], causal=causal, kv_lens=n, q_offsets=o if causal else None)
        seen = (pos[None, None] < n[:, None, None]).expand(-1, Nq, -1)
        if causal:
            seen = seen & (pos[None, None] <= o[:, None, None] + torch.arange(Nq, device="cuda")[None, :, None])
        kd, vd = (x[rows].double().repeat_interleave(Hq // Hkv, 1) for x in (k, v))
        s = (q[rows].double() @ kd.transpose(2, 3) / D ** 0.5).masked_fill(~seen[:, None], float("-inf"))
        ref = torch.softmax(s, -1) @ vd  # (NaN rows where nothing is visible, as a division by a zero sum gives)
        _check(out, lse, util.to_np(ref), util.to_np(torch.logsumexp(s, -1)))


@pytest.mark.skipif("RT_ATTN_PREFILL_F32_CLUSTER" in os.environ, reason="the child process itself")
@pytest.mark.parametrize("size", ["1", "2", "4", "8"])
def test_every_cluster_size(size):
    run_tests_with("RT_ATTN_PREFILL_F32_CLUSTER", size, "test_gpu_f32_cluster.py", "shared_row_blocks or without_a_visible or few_rows")
