"""The extension behind the device-tensor wrappers against the wrappers' own ctypes path: same results bit for bit,
and calls the extension does not cover (layouts to copy, invalid arguments) still reach that path."""
import pytest

pytestmark = pytest.mark.gpu


class _Nothing:
    """Stands in for the extension and covers nothing."""
    def __getattr__(self, name):
        return lambda *args: None


def _calls(torch, rt):
    g = torch.Generator(device="cuda").manual_seed(3)
    rn = lambda *s, dtype=torch.bfloat16: torch.randn(s, dtype=dtype, device="cuda", generator=g)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    q, k, v, do = (rn(2, 4, 130, 64) for _ in range(4))
    keep = torch.arange(130, device="cuda") % 3 != 1
    keep[0] = True
    f = [t.float() for t in (q, k, v, do)]
    out, lse = rt.prefill_bf16(q, k, v, causal=True)
    fout, flse = rt.prefill_f32(*f[:3], causal=True)
    qd, kc, vc = rn(2, 8, 128), rn(2, 2, 700, 128), rn(2, 2, 700, 128)
    act = [rn(2, 130, 4 * 64), rn(2, 130, 2 * 64), rn(2, 130, 2 * 64)]

    def rope():
        q2, k2, v2 = qd.clone(), kc.clone(), vc.clone()
        rt.rope_kv_append(q2, kc[:, :, 0].contiguous(), vc[:, :, 0].contiguous(), k2, v2, rt.rope_inv_freq(128),
                          positions=i32(5, 699))
        return q2, k2, v2

    return {
        "decode": lambda: rt.gqa_decode(qd, kc, vc, kv_lens=i32(700, 33)),
        "decode_f32_range": lambda: rt.gqa_decode(qd, kc, vc, kv_len=600, kv_begin=70, kv_end=500, scale=0.1,
                                                  out_dtype=torch.float32, return_lse=False),
        "rope": rope,
        "prefill": lambda: rt.prefill_bf16(q, k, v, causal=True, kv_lens=i32(130, 7)),
        "prefill_bool_keep": lambda: rt.prefill_bf16(q, k, v, key_keep=keep),
        "prefill_int_keep": lambda: rt.prefill_bf16(q, k, v, key_keep=keep.int()),  # converted by the wrapper
        "prefill_chunk": lambda: rt.prefill_bf16(q[:, :, :50].contiguous(), k, v, causal=True, q_offsets=i32(80, 3)),
        "prefill_strided": lambda: rt.prefill_bf16(*(t.transpose(1, 2) for t in (q, k, v)), scale=1),
        "mha": lambda: rt.mha_prefill_bf16(*act, 4, 2, causal=True),
        "mha_gap": lambda: rt.mha_prefill_bf16(act[0].repeat(1, 1, 2)[..., :256], *act[1:], 4, 2),  # not dense
        "f32": lambda: rt.prefill_f32(*f[:3], key_keep=keep),
        "backward_bf16": lambda: rt.backward_bf16(q, k, v, out, do, lse, causal=True),
        "backward_f32": lambda: rt.backward_f32(*f[:3], fout, f[3], flse, causal=True),
    }


@pytest.mark.parametrize("name", ["decode", "decode_f32_range", "rope", "prefill", "prefill_bool_keep", "prefill_int_keep",
                                  "prefill_chunk", "prefill_strided", "mha", "mha_gap", "f32", "backward_bf16", "backward_f32"])
def test_extension_and_ctypes_paths_agree(name, monkeypatch):
    import torch
    import rustorch_b200 as rt
    from rustorch_b200 import _lib
    call = _calls(torch, rt)[name]
    got = call()
    monkeypatch.setattr(_lib, "_binding", _Nothing())
    want = call()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype
            assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))


class _NoTruth:
    def __bool__(self):
        raise ValueError("truth is ambiguous")


@pytest.mark.parametrize("name", ["decode", "prefill", "prefill_lse", "mha", "mha_lse", "f32", "backward_bf16", "backward_f32"])
def test_flag_without_a_truth_value_raises_its_own_error(name):
    """A flag whose truth test raises (as an array of several elements does): the caller sees that error."""
    import torch
    import rustorch_b200 as rt
    x = torch.zeros(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16)
    f, act, qd = x.float(), x.view(1, 64, 128), x[:, :, 0].contiguous()
    lse, bad = torch.zeros(1, 2, 64, device="cuda"), _NoTruth()
    call = {
        "decode": lambda: rt.gqa_decode(qd, x, x, kv_len=3, return_lse=bad),
        "prefill": lambda: rt.prefill_bf16(x, x, x, causal=bad),
        "prefill_lse": lambda: rt.prefill_bf16(x, x, x, return_lse=bad),
        "mha": lambda: rt.mha_prefill_bf16(act, act, act, 2, causal=bad),
        "mha_lse": lambda: rt.mha_prefill_bf16(act, act, act, 2, return_lse=bad),
        "f32": lambda: rt.prefill_f32(f, f, f, causal=bad),
        "backward_bf16": lambda: rt.backward_bf16(x, x, x, x, x, lse, causal=bad),
        "backward_f32": lambda: rt.backward_f32(f, f, f, f, f, lse, causal=bad),
    }[name]
    with pytest.raises(ValueError, match="truth is ambiguous"):
        call()
