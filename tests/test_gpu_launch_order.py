"""Launches that overlap the one before them (programmatic stream serialization): each waits for it before it reads memory."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_backward_passes_on_one_workspace_with_changing_inputs(tt):
    """Few key/value heads: the dK/dV pass has 4 items and the dQ pass 128, so most SMs run the dQ pass of every step without
    having run its dK/dV pass.  Statistics and inputs change in place from step to step; steps queued back to back give the
    bits of steps that ran alone."""
    B, H, Hkv, S, D, steps = 1, 32, 1, 512, 128, 12
    g = torch.Generator(device="cuda").manual_seed(3)
    n = lambda h: torch.randn(steps, B, h, S, D, generator=g, device="cuda").bfloat16()
    qs, ks, vs, dos = n(H), n(Hkv), n(Hkv), n(H)
    alone = []
    for i in range(steps):
        out, lse = tt.attention_forward(qs[i], ks[i], vs[i], causal=True)
        torch.cuda.synchronize()
        alone.append((out, lse, *tt.attention_backward(qs[i], ks[i], vs[i], out, lse, dos[i], causal=True)))
        torch.cuda.synchronize()
    q, k, v, do = (torch.empty_like(t[0]) for t in (qs, ks, vs, dos))
    d = tt.capi.make_desc(B, H, S, S, D, tt.capi.TT_BF16, True, None, Hkv=Hkv)
    ws = torch.empty(int(tt.capi.lib.tt_attn_bwd_workspace_bytes(d)), dtype=torch.uint8, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(B, H, S, device="cuda")
    queued = []
    for i in range(steps):
        for dst, src in ((q, qs), (k, ks), (v, vs), (do, dos)):
            dst.copy_(src[i])
        tt.attention_forward(q, k, v, causal=True, out=out, lse=lse)
        grads = tt.attention_backward(q, k, v, out, lse, do, causal=True, workspace=ws)
        queued.append((out.clone(), lse.clone(), *grads))
    tt.check_device_status()
    for i in range(steps):
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), alone[i], queued[i]):
            assert torch.equal(a, b), (i, name)
