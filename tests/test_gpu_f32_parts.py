"""Float attention on the tensor cores (attn_f32_sm100.cu: three bf16 parts per value, tiles of 128 resident and 64 or 32
streamed rows) against the float64 closed form.

Bound: a product loses below 2^-23 to the terms left out, a tile's sum a few units of 2^-23 to truncating additions, and
tiles are added in float32; with the condition numbers of these inputs (sums of N(0,1) products) 2e-6 of the largest
element covers it, a fifth of the package's 1e-5 for float32.  The float64 reference makes the bound a statement about the
kernel alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
TOL = 2e-6


# head dims on both sides of the two tile widths and of the 8-value chunks; row counts around 32, 64 and 128; more keys than
# queries, one query, grouped heads, no mask and causal
@pytest.mark.parametrize("B,H,Hkv,S,L,D,causal", [
    (1, 1, 1, 1, 1, 4, False), (2, 2, 2, 64, 64, 32, False), (1, 2, 1, 65, 127, 64, True), (1, 2, 2, 128, 128, 64, False),
    (2, 4, 2, 129, 257, 60, True), (1, 2, 2, 33, 97, 68, True), (1, 4, 1, 160, 161, 128, True), (1, 2, 2, 1, 500, 128, False),
    (1, 1, 1, 700, 700, 64, True), (1, 2, 2, 300, 333, 100, False)])
def test_against_float64(tt, oracle, B, H, Hkv, S, L, D, causal):
    q, _, _, do = oracle.make_inputs(S + D, B, H, S, L, D)
    _, k, v, _ = oracle.make_inputs(S + D + 1, B, Hkv, S, L, D)
    ref = oracle.closed_form_f64(q, oracle.expand_kv_heads(k, H), oracle.expand_kv_heads(v, H), do, causal)
    tq, tk, tv, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, do))
    out, lse = tt.attention_forward(tq, tk, tv, causal=causal)
    dq, dk, dv = tt.attention_backward(tq, tk, tv, out, lse, tdo, causal=causal)
    tt.check_device_status()
    o_r, lse_r, dq_r, dk_r, dv_r = ref
    dk_r, dv_r = oracle.reduce_kv_heads(dk_r, Hkv), oracle.reduce_kv_heads(dv_r, Hkv)
    assert float(np.abs(lse.cpu().numpy() - lse_r).max()) <= 2e-6 * max(1.0, float(np.abs(lse_r).max()))
    for name, got, want in (("out", out, o_r), ("dq", dq, dq_r), ("dk", dk, dk_r), ("dv", dv, dv_r)):
        # one key: the softmax gradient is zero and only rounding is left of dq and dk; measure those against |dO||k|
        scale = max(float(np.abs(want).max()), 1.0)
        assert float(np.abs(got.cpu().numpy() - want).max()) <= TOL * scale, name


@pytest.mark.parametrize("D,lens", [(64, [1, 64, 65, 200]), (128, [31, 33, 128, 129])])
def test_padded_keys(tt, oracle, D, lens):
    """Keys behind a length take no part, whatever finite values they hold, and get zero gradients."""
    B, H, S, L = len(lens), 2, 70, 200
    q, k, v, do = oracle.make_inputs(D, B, H, S, L, D)
    for b, n in enumerate(lens):
        k[b, :, n:] = 1e30
        v[b, :, n:] = -1e30
    tq, tk, tv, tdo = (torch.from_numpy(x).cuda() for x in (q, k, v, do))
    tl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out, lse = tt.attention_forward(tq, tk, tv, kv_lens=tl)
    dq, dk, dv = tt.attention_backward(tq, tk, tv, out, lse, tdo, kv_lens=tl)
    tt.check_device_status()
    for b, n in enumerate(lens):
        o_r, _, dq_r, dk_r, dv_r = oracle.closed_form_f64(q[b:b + 1], k[b:b + 1, :, :n], v[b:b + 1, :, :n], do[b:b + 1], False)
        for name, got, want in (("out", out[b:b + 1], o_r), ("dq", dq[b:b + 1], dq_r), ("dk", dk[b:b + 1, :, :n], dk_r),
                                ("dv", dv[b:b + 1, :, :n], dv_r)):
            assert float(np.abs(got.cpu().numpy() - want).max()) <= TOL * max(float(np.abs(want).max()), 1.0), (name, n)
        assert float(dk[b, :, n:].abs().max() if n < L else 0.0) == 0.0 and float(dv[b, :, n:].abs().max() if n < L else 0.0) == 0.0


def test_largest_finite_values(tt, oracle):
    """A value next to the largest float keeps its size (its first bf16 part must not round to infinity), and takes no part
    in the rows that the mask hides it from."""
    S, D = 150, 64
    q, k, v, _ = oracle.make_inputs(5, 1, 1, S, S, D)
    big = np.finfo(np.float32).max
    want = oracle.closed_form_f64(q, k, v, np.zeros_like(q), True)[0]
    v[0, 0, S - 1] = -big
    out, _ = tt.attention_forward(*(torch.from_numpy(x).cuda() for x in (q, k, v)), causal=True)
    tt.check_device_status()
    got = out.cpu().numpy()
    assert float(np.abs(got[:, :, :S - 1] - want[:, :, :S - 1]).max()) <= TOL * max(float(np.abs(want).max()), 1.0)
    s = (q[0, 0, S - 1].astype(np.float64) @ k[0, 0].T.astype(np.float64)) / np.sqrt(D)
    p = np.exp(s - s.max())
    last = -(p / p.sum())[S - 1] * float(big)
    assert float(np.abs(got[0, 0, S - 1] / last - 1).max()) <= 1e-5
