"""The bf16 backward where a tile of the other side holds one 64-row step or two and a CTA works through several items
(csrc/backward_tcgen05.cu: the statistics' slots, score buffers and ring phases run on from item to item)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("N", [1, 63, 64, 65, 128, 129, 192, 193, 257])
def test_items_of_few_steps(N, causal, D):
    """Bit for bit what each sequence gives on its own, and torch in f32 to the limit of bf16 products."""
    import torch
    import rustorch_b200 as rt
    B, H = 8, 60
    torch.manual_seed(N)
    q, k, v, do = (torch.randn(B, H, N, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    out, lse = rt.prefill_bf16(q, k, v, causal=causal)
    grads = rt.backward_bf16(q, k, v, out, do, lse, causal=causal)
    for b in (0, B - 1):
        s = slice(b, b + 1)
        for whole, piece in zip(grads, rt.backward_bf16(*(x[s].contiguous() for x in (q, k, v, out, do, lse)), causal=causal)):
            assert torch.equal(whole[s], piece)
    x = [t.float().requires_grad_() for t in (q, k, v)]
    w = x[0] @ x[1].transpose(2, 3) / D ** 0.5
    if causal:
        w = w.masked_fill(torch.ones(N, N, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    (torch.softmax(w, -1) @ x[2]).backward(do.float())
    for g, r in zip(grads, x):
        # P and dS are rounded to bf16 (2^-9 each); with one visible key dQ and dK are rounding noise around zero
        assert float((g - r.grad).norm()) <= 1e-2 * float(r.grad.norm()) + 4e-3 * (B * H * D) ** 0.5
