"""The f32 tiles have a pitch of their kernel's widest head dim (csrc/simt_tile.cuh): head dims at both ends of every width, after
a launch that leaves NaN in the columns which these do not fill, against the CPU oracle at the f32 kernels' own gates."""
import numpy as np
import pytest

from tests import util
from tests.test_gpu_backward import _check, _det, _gpu_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 3, 31, 32, 33, 62, 64, 65, 96, 97, 126, 128, 129, 200, 255, 256])
@pytest.mark.parametrize("causal", [False, True])
def test_columns_beyond_the_head_dim(oracle, D, causal):
    import torch
    import rustorch_b200 as rt
    full = 256 if D > 128 else (D + 31) // 32 * 32
    nan = torch.full((8, 37, 64, full), float("nan"), device="cuda")  # two CTAs per SM, one after the other
    o, lse = rt.prefill_f32(nan, nan, nan)
    rt.backward_f32(nan, nan, nan, o, nan, lse)
    q, k, v, do_ = (_det(oracle, (1, 3, 150, D), s) for s in (1, 2, 3, 4))
    out, lse = rt.prefill_f32(*(util.to_cuda(x) for x in (q, k, v)), causal=causal)
    _, ref, ref_lse = oracle.flash_forward_ext(q, k, v, causal=causal)
    assert np.abs(util.to_np(out) - ref).max() < 1e-4 and np.abs(util.to_np(lse) - ref_lse).max() < 1e-4
    rc, *refs = oracle.flash_backward(q, k, v, do_, causal=causal)
    assert rc == 0
    for name, got, want in zip(("dq", "dk", "dv"), _gpu_backward(q, k, v, do_, causal), refs):
        _check(got, want, f"{name} D={D} causal={causal}")
