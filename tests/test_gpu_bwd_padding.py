"""Key tiles that are all padding: the backward reads nothing of them, so finite padding whose products overflow stays out of dq."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["fused", "two_pass"])
@pytest.mark.parametrize("H,Hkv,S,L,D,lens,causal", [
    (2, 2, 300, 640, 128, [128, 640, 384], False),
    (4, 2, 130, 384, 64, [256, 128, 384], False),
    (1, 1, 384, 384, 128, [128, 256, 384], True),
    (8, 8, 257, 1500, 64, [128] * 20, False),      # more padded tiles than SMs: a CTA passes over several in a row
    (2, 2, 200, 200, 128, [1, 128, 200], False),   # a boundary inside a tile beside one at its end
])
def test_padded_tiles_are_not_read(tt, oracle, monkeypatch, path, H, Hkv, S, L, D, lens, causal):
    monkeypatch.setenv("TT_BWD_PATH", path)
    B = len(lens)
    q, _, _, do = (None if x is None else oracle.bf16_round(x) for x in oracle.make_inputs(61, B, H, S, L, D, sigma=0.6))
    _, k, v, _ = (None if x is None else oracle.bf16_round(x) for x in oracle.make_inputs(62, B, Hkv, S, L, D, sigma=0.6))
    dev = lambda x: torch.from_numpy(x).to("cuda", dtype=torch.bfloat16)
    tq, tk, tv, tdo = (dev(x) for x in (q, k, v, do))
    for b, n in enumerate(lens):
        whole = -(-n // 128) * 128               # from here on no tile has a key that counts
        tk[b, :, n:], tv[b, :, n:] = 0.0, 0.0
        tv[b, :, whole:] = 3e38                  # dO V overflows
    tl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out, lse = tt.attention_forward(tq, tk, tv, causal=causal, kv_lens=tl)
    grads = tt.attention_backward(tq, tk, tv, out, lse, tdo, causal=causal, kv_lens=tl)
    tt.check_device_status()
    f = lambda t: t.float().cpu().numpy()
    for b, n in enumerate(lens):
        if causal and n < L:
            assert all(bool(torch.isfinite(g[b].float()).all()) for g in grads)
        else:
            _, _, *want = oracle.attention_backward_grouped(q[b:b + 1], k[b:b + 1, :, :n], v[b:b + 1, :, :n], do[b:b + 1], causal)
            for name, got, ref in zip(("dq", "dk", "dv"), grads, want):
                got = f(got[b:b + 1] if name == "dq" else got[b:b + 1, :, :n])
                assert oracle.max_abs_err(got, ref) <= oracle.bf16_grad_tol(ref), name
        assert not grads[1][b, :, n:].any() and not grads[2][b, :, n:].any()
