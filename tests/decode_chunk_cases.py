"""Where a decode launch cuts the sequences under RT_ATTN_DECODE_CHUNK.  The library reads the variable once per process:
tests/test_gpu_overrides.py runs this file in a child process with it set."""
import os

import numpy as np
import pytest

from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,D,S,lens", [
    (1, 8, 2, 128, 1000, None),            # one sequence
    (3, 16, 8, 128, 4096, (1, 4096)),      # a batch that is cut into shares without the override
    (40, 16, 8, 128, 500, (500, 65)),      # and ones that are left whole
    (2, 8, 1, 256, 2100, (2050, 2099)),    # or cut into equal parts
])
def test_every_sequence_is_cut_at_the_given_length(oracle, B, Hq, Hkv, D, S, lens):
    """The scratch holds one log-sum-exp per chunk and row: that of exactly the chunk's tokens."""
    import torch
    import rustorch_b200 as rt
    chunk = int(os.environ["RT_ATTN_DECODE_CHUNK"])
    r = np.random.default_rng(9)
    n = np.full(B, S, dtype=np.int32) if lens is None else r.integers(min(lens), max(lens) + 1, B).astype(np.int32)
    if lens:
        n[0], n[-1] = lens
    q = util.normal_bf16(oracle, (B, Hq, D), 1)
    k, v = (util.normal_bf16(oracle, (B, Hkv, S, D), s) for s in (2, 3))
    t = [util.to_cuda_bf16(x) for x in (q, k, v)]
    parts = -(-S // chunk)
    need = rt.decode_workspace_bytes(B, Hq, Hkv, D, S)
    assert need >= parts * B * Hq * (D + 1) * 4
    ws = torch.full((need,), 0xff, dtype=torch.uint8, device="cuda")  # NaN wherever nothing is written
    out, lse = rt.gqa_decode(*t, kv_lens=None if lens is None else util.to_cuda(n), kv_len=S if lens is None else None, workspace=ws)
    torch.cuda.synchronize()
    _, ref, ref_lse = oracle.gqa_decode_cache(q, k, v, n)
    util.check_output(util.to_np(out), ref)
    util.check_lse(util.to_np(lse), ref_lse)
    at = parts * B * Hq * D
    got = ws.view(torch.float32)[at:at + parts * B * Hq].cpu().numpy().reshape(parts, B, Hq)
    s = np.einsum("bhgd,bhsd->bhgs", q.reshape(B, Hkv, Hq // Hkv, D), k) / np.sqrt(D)
    s = s.reshape(B, Hq, S)
    s[np.arange(S)[None, None, :] >= n[:, None, None].repeat(Hq, 1)] = -np.inf
    with np.errstate(divide="ignore"):
        want = np.stack([np.log(np.exp(s[..., c:c + chunk]).sum(-1)) for c in range(0, S, chunk)])
    util.check_lse(got, want)
