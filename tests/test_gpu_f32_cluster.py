"""The f32 forward where a cluster of CTAs shares the keys of a row block (csrc/prefill_simt.cu, kSplit): launches of few row blocks,
keys at the edges of a CTA's share of 64-key tiles, against the CPU oracle at the f32 kernels' 1e-4."""
import numpy as np
import pytest

from tests import util

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
