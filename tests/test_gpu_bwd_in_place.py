"""dk and dv written over k and v, at head dim 64: every item of the single pass reads its keys ahead of writing their gradients."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hkv,S,L,causal", [(1, 2, 2, 300, 300, True), (2, 8, 2, 129, 700, False), (2, 16, 16, 1024, 1024, True)])
def test_gradients_over_keys_and_values(tt, B, H, Hkv, S, L, causal):
    tt.set_backward_deterministic(False)
    g = torch.Generator(device="cuda").manual_seed(L)
    n = lambda h, s: torch.randn(B, h, s, 64, generator=g, device="cuda").bfloat16()
    q, k, v, do = n(H, S), n(Hkv, L), n(Hkv, L), n(H, S)
    out, lse = tt.attention_forward(q, k, v, causal=causal)
    want = tt.attention_backward(q, k, v, out, lse, do, causal=causal)
    d = tt.capi.make_desc(B, H, S, L, 64, tt.capi.TT_BF16, causal, None, Hkv=Hkv)
    lib, p = tt.capi.lib, lambda t: ctypes.c_void_p(t.data_ptr())
    need = int(lib.tt_attn_bwd_workspace_bytes(ctypes.byref(d)))
    ws, dq = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.empty_like(q)
    tt.capi.check(lib.tt_attn_bwd(ctypes.byref(d), p(q), p(k), p(v), p(out), p(lse), p(do), p(dq), p(k), p(v), p(ws), need,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    tt.check_device_status()
    for name, a, b in zip(("dq", "dk", "dv"), (dq, k, v), want):   # one step of bf16: the sums' order may differ
        assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * float(b.float().abs().max()), name
