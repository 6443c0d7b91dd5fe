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


def names_of(tt, call):
    tt.capi.profile_enable(True)
    tt.capi.profile_reset()
    r = call()
    ran = set(tt.capi.profile_read())
    tt.capi.profile_enable(False)
    return r, ran


def in_one_launch(key_tiles):
    return 5 * key_tiles <= 9 * torch.cuda.get_device_properties(0).multi_processor_count


# both passes of the two-pass backward in one launch, up to 1.8 items per SM in the first: one item, one and two waves of each,
# both sides of the limit (266 on 148 SMs), tails, grouped heads; head dim 64 where its two passes are asked for
@pytest.mark.parametrize("B,H,Hkv,S,L,D,causal", [(1, 1, 1, 1, 1, 128, False), (1, 4, 2, 130, 515, 128, True), (1, 37, 37, 512, 512, 128, True), (1, 148, 4, 128, 300, 128, True),
                                                  (1, 1, 1, 100, 266 * 128, 128, False), (1, 1, 1, 100, 266 * 128 + 1, 128, False), (1, 300, 1, 128, 128, 128, False),
                                                  (1, 37, 37, 640, 640, 128, True), (2, 8, 2, 500, 600, 64, True)])
def test_two_passes_in_one_launch(tt, oracle, monkeypatch, B, H, Hkv, S, L, D, causal):
    monkeypatch.setenv("TT_BWD_PATH", "two_pass")
    q, _, _, do = oracle.make_inputs(S + D, B, H, S, L, D)
    _, k, v, _ = oracle.make_inputs(S + D + 1, B, Hkv, S, L, D)
    q, k, v, do = (oracle.bf16_round(a) for a in (q, k, v, do))
    tq, tk, tv, tdo = (torch.from_numpy(a).cuda().bfloat16() for a in (q, k, v, do))
    out, lse = tt.attention_forward(tq, tk, tv, causal=causal)
    (dq, dk, dv), ran = names_of(tt, lambda: tt.attention_backward(tq, tk, tv, out, lse, tdo, causal=causal))
    tt.check_device_status()
    assert ran == {"attn_bwd_prep"} | ({"attn_bwd_sm100_both"} if in_one_launch(B * Hkv * -(-L // 128)) else {"attn_bwd_sm100_dkv", "attn_bwd_sm100_dq"})
    _, _, dq_r, dk_r, dv_r = oracle.attention_backward_grouped(q, k, v, do, causal)
    for name, got, ref in (("dq", dq, dq_r), ("dk", dk, dk_r), ("dv", dv, dv_r)):
        assert oracle.max_abs_err(got.float().cpu().numpy(), ref) <= oracle.bf16_grad_tol(ref), name


def test_packed_passes_in_one_launch(tt, oracle):
    """Sequences of a packed batch equal dense calls, in one launch or (long batches) two, to the bit."""
    H, Hkv, D = 4, 2, 128
    for lens in ([1, 130, 257, 64], [1, 700, 1300, 64, 500, 900, 20, 1000, 128, 300, 777, 1], [300] * 70):
        total, cu = sum(lens), torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(len(lens))
        n = lambda h: torch.randn(total, h, D, generator=g, device="cuda").bfloat16()
        q, do, k, v = n(H), n(H), n(Hkv), n(Hkv)
        m = max(lens)
        out, lse = tt.attention_forward_varlen(q, k, v, cu, cu, m, m, causal=True)
        grads, ran = names_of(tt, lambda: tt.attention_backward_varlen(q, k, v, cu, cu, m, m, out, lse, do, causal=True))
        assert ("attn_bwd_sm100_both" in ran) == in_one_launch(len(lens) * Hkv * -(-m // 128))
        for i, s in enumerate(lens):
            rows = slice(sum(lens[:i]), sum(lens[:i]) + s)
            dense = [t[rows].transpose(0, 1)[None].contiguous() for t in (q, k, v, do)]
            o, l = tt.attention_forward(*dense[:3], causal=True)
            want = tt.attention_backward(*dense[:3], o, l, dense[3], causal=True)
            for a, b in zip(grads, want):
                assert torch.equal(a[rows].transpose(0, 1)[None], b)
    tt.check_device_status()


@pytest.mark.parametrize("shared", ["q", "dout"])
@pytest.mark.parametrize("S", [256, 2176])   # (two launches by the rule: 272 tiles)
def test_dq_over_an_input_of_the_c_call(tt, shared, S):
    """The dQ pass comes last, so a caller of the C ABI may give it q's or dout's memory."""
    import ctypes
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, do = (torch.randn(1, 16, S, 128, generator=g, device="cuda").bfloat16() for _ in range(4))
    out, lse = tt.attention_forward(q, k, v, causal=True)
    want = tt.attention_backward(q, k, v, out, lse, do, causal=True)
    d = tt.capi.make_desc(1, 16, S, S, 128, tt.capi.TT_BF16, True)
    n = int(tt.capi.lib.tt_attn_bwd_workspace_bytes(ctypes.byref(d)))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    dq = q if shared == "q" else do
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    tt.capi.check(tt.capi.lib.tt_attn_bwd(ctypes.byref(d), p(q), p(k), p(v), p(out), p(lse), p(do), p(dq), p(dk), p(dv), p(ws), n,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    tt.check_device_status()
    for a, b in zip((dq, dk, dv), want):
        assert torch.equal(a, b)
