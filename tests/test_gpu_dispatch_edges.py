"""Sizes at which a branch of a kernel or of a launch rule changes, each against the CPU oracle or, where that would take
minutes (schedules, sorted keep flags, clusters), against torch in f32 to the same limits."""
import numpy as np
import pytest

from tests import util
from tests.test_gpu_prefill_tc import _qkv, _run_tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N,causal", [(1, False), (65, True), (129, False), (321, True), (650, False)])
def test_keep_flags_with_hidden_tails(oracle, D, N, causal):
    """Keep flags whose last kept key sits on either side of a 64- and a 128-key step, holes between, and a row of
    flags that keeps nothing (NaN rows, LSE -inf)."""
    kept = [n for n in (0, 1, 63, 64, 65, 128, 129, N) if n <= N]
    keep = np.zeros((len(kept), N), dtype=np.uint8)
    for b, n in enumerate(kept):
        keep[b, :n] = 1
        keep[b, 3:max(3, n - 1):5] = 0
    q, k, v = _qkv(oracle, (len(kept), 2, N, D))
    out, lse = _run_tc(q, k, v, causal=causal, key_keep=util.to_cuda(keep))
    _, ref, ref_lse = oracle.flash_forward_ext(q, k, v, causal=causal, keep=keep)
    util.check_output(out, ref, label=f"keep tails N{N} D{D} causal={causal}")
    util.check_lse(lse, ref_lse)


@pytest.mark.parametrize("N", [1, 17, 64, 65, 130, 200])
@pytest.mark.parametrize("D", [1, 7, 32, 33, 64, 80, 96, 100, 128, 129, 200, 256])
def test_f32_forward_and_backward_tiles(oracle, N, D):
    """The register-tiled f32 kernels where their tiles, column groups, 16-byte copies and two-group split end."""
    import torch
    import rustorch_b200 as rt
    for causal in (False, True):
        q, k, v, do = (oracle.fill_normal((1, 2, N, D), s) for s in (1, 2, 3, 4))
        t = [util.to_cuda(x) for x in (q, k, v, do)]
        out, lse = rt.prefill_f32(*t[:3], causal=causal)
        got = rt.backward_f32(*t[:3], out, t[3], lse, causal=causal)
        torch.cuda.synchronize()
        _, ref, ref_lse = oracle.flash_forward_ext(q, k, v, causal=causal)
        assert np.abs(util.to_np(out) - ref).max() < 1e-4
        assert np.abs(util.to_np(lse) - ref_lse).max() < 1e-4
        _, *grads = oracle.flash_backward(q, k, v, do, causal=causal)
        for name, a, b in zip(("dq", "dk", "dv"), got, grads):
            assert np.abs(util.to_np(a) - b).max() < 2e-4 * max(1.0, np.abs(b).max()), (name, causal)


@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("B,H,N", [(1, 1, 1), (1, 2, 300), (3, 5, 1000), (1, 40, 2100)])
def test_host_entry_staged_equals_pinned(precision, B, H, N):
    """Pageable slices (staging threads, conversion on the host) and pinned ones (copied as they are, conversion on
    the device) give the same result: one piece, several chunks, and more pieces than the ring has slots.  The inputs
    hold values whose bf16 rounding is special.  (Chunks of another size may split the keys of a bf16 launch another
    way, which moves last bits; the f32 kernels have one order.)"""
    def same(a, b):
        if precision == "f32":
            return np.array_equal(a.view(np.uint32), b.view(np.uint32))
        return np.allclose(a, b, rtol=1e-2, atol=1e-2)
    import torch
    import rustorch_b200 as rt
    D, n = 64, B * H * N * 64
    r = np.random.default_rng(7)
    q, k, v = (r.standard_normal(n, dtype=np.float32) for _ in range(3))
    v[:10] = [1.00390625, 1.01171875, -0.0, 1e-40, 3e38, -1.0, 65504.0, 1e-30, 0.99609375, 2.0]
    shape, mask = rt.AttentionShape.new(B, H, N, D), rt.Mask.causal()
    out = np.empty_like(q)
    rt.flash_forward_masked(shape, q, k, v, mask, out, precision)
    pinned = [torch.empty(n, dtype=torch.float32, pin_memory=True).numpy() for _ in range(4)]
    for p, x in zip(pinned, (q, k, v)):
        p[:] = x
    rt.flash_forward_masked(shape, *pinned[:3], mask, pinned[3], precision)
    assert same(out, pinned[3])
    mixed = np.empty_like(q)
    rt.flash_forward_masked(shape, q, pinned[1], v, mask, mixed, precision)
    assert same(out, mixed)


@pytest.mark.parametrize("B,Hq,Hkv,D,S,lens", [
    (40, 16, 8, 128, 200, (0, 200)),      # at least as many groups as CTAs: whole sequences
    (40, 8, 8, 64, 300, (1, 300)),        # 64 groups and more, little each: whole
    (3, 16, 8, 128, 4096, (0, 4096)),     # shares of all tokens, one sequence empty
    (32, 4, 2, 64, 2600, (5, 2600)),      # the same with a full warp of sequences
    (2, 8, 1, 256, 2100, (2050, 2099)),   # equal parts of every sequence
    (33, 8, 2, 128, 2300, (0, 2300)),     # the same with more sequences than a warp has lanes
    (37, 4, 4, 64, 2400, (0, 2400)),      # and merged by the CTA that completes a group
    (5, 4, 2, 128, 1000, (63, 65)),       # fixed parts, most of them empty
    (1, 4, 1, 64, 40000, (39999, 39999)),  # one group: as many parts as its merge is worth
    (90, 1, 1, 256, 1100, (900, 1100)),   # D = 256: two waves
])
def test_decode_splits(oracle, B, Hq, Hkv, D, S, lens):
    """One launch of each rule of the decode split, with lengths at the ends of its range, whole and as a KV range."""
    import torch
    import rustorch_b200 as rt
    r = np.random.default_rng(5)
    n = r.integers(lens[0], lens[1] + 1, B).astype(np.int32)
    n[0], n[-1] = lens
    q = util.normal_bf16(oracle, (B, Hq, D), 1)
    k, v = (util.normal_bf16(oracle, (B, Hkv, S, D), s) for s in (2, 3))
    dq, dk, dv, dn = *(util.to_cuda_bf16(x) for x in (q, k, v)), util.to_cuda(n)
    out, lse = rt.gqa_decode(dq, dk, dv, kv_lens=dn)
    torch.cuda.synchronize()
    _, ref, ref_lse = oracle.gqa_decode_cache(q, k, v, n)
    util.check_output(util.to_np(out), ref, label="whole")
    util.check_lse(util.to_np(lse), ref_lse)
    cut = S // 3
    parts = [rt.gqa_decode(dq, dk, dv, kv_lens=dn, kv_begin=a, kv_end=b, out_dtype=torch.float32)
             for a, b in ((0, cut), (cut, S))]
    out, lse = rt.merge_partials(torch.stack([p[0].reshape(B * Hq, D) for p in parts]),
                                 torch.stack([p[1].reshape(B * Hq) for p in parts]))
    util.check_output(util.to_np(out).reshape(B, Hq, D), ref, label="range")
    util.check_lse(util.to_np(lse).reshape(B, Hq), ref_lse)


@pytest.mark.parametrize("B,H,N,D,causal,part", [
    (28, 20, 1200, 64, True, 7),     # more K/V than L2: paired rounds that end inside a head, levels for the rest
    (26, 16, 1100, 128, True, 13),   # the same, last tile of a head without rows
    (12, 16, 300, 64, True, 4),      # levels only; the parts fall below one item per SM
    (20, 16, 777, 64, False, 5),     # head after head, ragged blocks last
    (3, 50, 130, 128, False, 3),     # one block more than SMs
    (6, 16, 1000, 128, True, 2),     # the parts: more 128-row items than SMs, by levels
    (4, 16, 100, 64, True, 1),       # one ragged 128-row item per head
])
def test_prefill_schedules(B, H, N, D, causal, part):
    """Every block is visited once whatever the schedule: a launch gives what launches over parts of its batch give."""
    import torch
    import rustorch_b200 as rt
    torch.manual_seed(3)
    q, k, v = (torch.randn(B, H, N, D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    out, lse = rt.prefill_bf16(q, k, v, causal=causal)
    for b in range(0, B, part):
        o, l = rt.prefill_bf16(*(x[b:b + part] for x in (q, k, v)), causal=causal)
        assert torch.allclose(out[b:b + part].float(), o.float(), rtol=1e-2, atol=1e-2)
        assert torch.allclose(lse[b:b + part], l, rtol=1e-5, atol=1e-4)
    s = q[-1].float() @ k[-1].float().transpose(1, 2) / D ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(N, N, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = torch.softmax(s, -1) @ v[-1].float()
    assert float((out[-1].float() - ref).norm() / ref.norm()) <= util.TOL_REL_L2
    assert torch.allclose(lse[-1], torch.logsumexp(s, -1), rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("B,H,N,Nkv,D,causal", [(9, 12, 600, 600, 64, False), (9, 12, 600, 600, 128, True),
                                                 (6, 30, 200, 9000, 64, False), (13, 12, 257, 300, 128, False)])
def test_keep_flags_sorted(B, H, N, Nkv, D, causal):
    """Keep flags in the sorted schedule (tails of every length, beyond the searched 4096 keys too, holes, nothing kept)."""
    import torch
    import rustorch_b200 as rt
    torch.manual_seed(4)
    q = torch.randn(B, H, N, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, H, Nkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    keep = torch.ones(B, Nkv, device="cuda", dtype=torch.uint8)
    for b, hidden in enumerate([0, 1, 64, Nkv - 1, 300, Nkv // 2][:B]):
        keep[b, Nkv - hidden:] = 0
    keep[1, 5:90] = 0
    keep[2] = 0
    out, lse = rt.prefill_bf16(q, k, v, causal=causal, key_keep=keep)
    for b in range(B):
        s = q[b].float() @ k[b].float().transpose(1, 2) / D ** 0.5
        s = s.masked_fill(keep[b] == 0, float("-inf"))
        if causal:
            s = s.masked_fill(torch.ones(N, Nkv, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        ref = torch.softmax(s, -1) @ v[b].float()
        dead = torch.isinf(s).all(-1)
        assert torch.equal(torch.isnan(out[b]).all(-1), dead) and torch.equal(lse[b] == float("-inf"), dead)
        x, y = out[b].float()[~dead], ref[~dead]
        assert float((x - y).norm()) <= util.TOL_REL_L2 * float(y.norm())
        assert torch.allclose(lse[b][~dead], torch.logsumexp(s, -1)[~dead], rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nkv,D,causal,lens", [
    (1, 4, 2, 100, 9000, 64, True, (9000,)),          # 8 CTAs an item
    (2, 16, 2, 123, 8400, 128, True, (2100, 8400)),   # 4, one sequence much shorter
    (1, 33, 33, 1, 3000, 128, False, (2999,)),        # 4, as many clusters as fit
    (1, 74, 37, 128, 4097, 64, False, (4097,)),       # 2
    (3, 8, 8, 200, 5000, 128, False, (0, 1, 5000)),   # shares without a key, and a sequence without one
    (5, 4, 2, 70, 3000, 64, True, (70, 128, 129, 1500, 3000)),
])
def test_prefill_clusters(B, Hq, Hkv, Nq, Nkv, D, causal, lens):
    """Items whose keys a cluster of CTAs shares."""
    import torch
    import rustorch_b200 as rt
    torch.manual_seed(6)
    q = torch.randn(B, Hq, Nq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, Hkv, Nkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    n = torch.tensor(lens, device="cuda", dtype=torch.int32)
    off = torch.tensor([max(0, x - Nq) for x in lens], device="cuda", dtype=torch.int32)
    out, lse = rt.prefill_bf16(q, k, v, causal=causal, kv_lens=n, q_offsets=off if causal else None)
    for b in range(B):
        if lens[b] == 0:
            assert bool(torch.isnan(out[b]).all()) and bool((lse[b] == float("-inf")).all())
            continue
        kb, vb = (x[b, :, :lens[b]].float().repeat_interleave(Hq // Hkv, 0) for x in (k, v))
        s = q[b].float() @ kb.transpose(1, 2) / D ** 0.5
        if causal:
            s = s.masked_fill(torch.ones(Nq, lens[b], dtype=torch.bool, device="cuda").triu(int(off[b]) + 1), float("-inf"))
        ref = torch.softmax(s, -1) @ vb
        assert float((out[b].float() - ref).norm() / ref.norm()) <= util.TOL_REL_L2
        assert torch.allclose(lse[b], torch.logsumexp(s, -1), rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nkv,D,causal,lens", [
    (4, 16, 2, 300, 2500, 64, True, (300, 2500, 0, 2499)),   # one sequence empty, two alike
    (5, 8, 8, 513, 2600, 128, True, (640, 2600, 700, 513, 200)),  # fewer keys than queries: rows without a key
    (2, 40, 8, 200, 3000, 128, False, (129, 2999)),          # no mask: the length alone
    (32, 2, 1, 500, 4000, 64, True, (500, 4000)),            # as many pairs as are ranked
    (33, 2, 1, 500, 4000, 64, True, (500, 4000)),            # more: the order of the batch
])
def test_prefill_chunks_by_length(oracle, B, Hq, Hkv, Nq, Nkv, D, causal, lens):
    """More 128-row items than SMs, of sequences whose lengths only the device knows."""
    import rustorch_b200 as rt
    n = np.linspace(min(lens), max(lens), B).astype(np.int32) if len(lens) != B else np.array(lens, dtype=np.int32)
    if len(lens) != B:
        np.random.default_rng(2).shuffle(n)
    off = (n - Nq).astype(np.int32)
    q = util.normal_bf16(oracle, (B, Hq, Nq, D), util.SEED_Q)
    k, v = (util.normal_bf16(oracle, (B, Hkv, Nkv, D), s) for s in (util.SEED_K, util.SEED_V))
    out, lse = rt.prefill_bf16(*(util.to_cuda_bf16(x) for x in (q, k, v)), causal=causal, kv_lens=util.to_cuda(n),
                               q_offsets=util.to_cuda(off) if causal else None)
    _, ref, ref_lse = oracle.attention_general(q, k, v, causal=causal, kv_lens=n, q_offsets=off if causal else None)
    util.check_output(util.to_np(out), ref, label=f"B{B} {Nq}/{Nkv} D{D}")
    util.check_lse(util.to_np(lse), ref_lse)


@pytest.mark.parametrize("B,H,N,D,causal,part", [
    (2, 37, 129, 64, True, 1),      # as many tiles of both sides as SMs, then twice that
    (3, 64, 200, 64, False, 1),     # several tiles a CTA, an odd count of steps
    (28, 20, 1100, 64, True, 7),    # operands beyond L2: paired rounds that end inside a head
    (9, 16, 577, 128, True, 3),     # levels only, last tile with one row
])
def test_backward_schedules(B, H, N, D, causal, part):
    """Every tile of either side is visited once whatever the schedule: bit for bit what launches over parts of the
    batch give."""
    import torch
    import rustorch_b200 as rt
    torch.manual_seed(8)
    q, k, v, do = (torch.randn(B, H, N, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    out, lse = rt.prefill_bf16(q, k, v, causal=causal)
    grads = rt.backward_bf16(q, k, v, out, do, lse, causal=causal)
    for b in range(0, B, part):
        s = slice(b, b + part)
        for whole, piece in zip(grads, rt.backward_bf16(*(x[s].contiguous() for x in (q, k, v, out, do, lse)), causal=causal)):
            assert torch.equal(whole[s], piece)
    x = [t[-1].float().requires_grad_() for t in (q, k, v)]
    w = x[0] @ x[1].transpose(1, 2) / D ** 0.5
    if causal:
        w = w.masked_fill(torch.ones(N, N, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    (torch.softmax(w, -1) @ x[2]).backward(do[-1].float())
    for g, r in zip(grads, x):
        assert float((g[-1] - r.grad).norm() / r.grad.norm()) <= 1e-2
