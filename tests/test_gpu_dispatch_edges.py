"""Sizes at which a branch of a kernel or of a launch rule changes, each against the CPU oracle."""
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
