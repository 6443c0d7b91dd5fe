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


def visible_f32(q, k, v, do):
    """One slice, causal, in float32 over the pairs that the mask leaves: what it hides takes no part, not even as 0 x infinity."""
    S, D = q.shape
    scale = np.float32(1 / np.sqrt(D))
    out, lse, dq, dk, dv = np.zeros_like(q), np.zeros(S, np.float32), np.zeros_like(q), np.zeros_like(k), np.zeros_like(v)
    with np.errstate(all="ignore"):
        for i in range(S):
            K, V = k[:i + 1], v[:i + 1]
            s = (K * q[i]).sum(1) * scale
            m = np.fmax.reduce(s)
            e = np.exp(s - m)
            p = e / e.sum()
            lse[i], out[i] = m + np.log(e.sum()), (p[:, None] * V).sum(0)
            ds = p * ((V * do[i]).sum(1) - (out[i] * do[i]).sum())
            dq[i] = (ds[:, None] * K).sum(0) * scale
            dk[:i + 1] += ds[:, None] * q[i] * scale
            dv[:i + 1] += p[:, None] * do[i]
    return out, lse, dq, dk, dv


inf, nan = float("inf"), float("nan")


# an infinity or a NaN in each input; an infinity behind what early rows see; scores that overflow to -infinity (weight 0), from an
# infinity and from finite factors, and to +infinity; a product of finite gradients that overflows; a first part that rounds up
# (1.0039) and one that does not, because the signs of the cross terms come from the remainders
@pytest.mark.parametrize("D", [64, 128, 40])
@pytest.mark.parametrize("name,row,value", [("q", 9, inf), ("k", 150, inf), ("v", 150, inf), ("do", 150, -inf), ("q", 130, nan), ("k", 3, nan),
                                            ("v", 199, nan), ("do", 0, nan), ("k", 3, -inf), ("k", 150, -3e38), ("k", 7, 1.0039e30),
                                            ("k", 7, 1.0009e30), ("do", 60, 1.0039e38)])
def test_infinities_nan_and_overflow(tt, oracle, D, name, row, value):
    S = 200
    x = dict(zip(("q", "k", "v", "do"), (a[0, 0] for a in oracle.make_inputs(D, 1, 1, S, S, D))))
    if name == "k" and not np.isnan(value):
        x["q"] = np.abs(x["q"]) + np.float32(0.5)       # scores of that key have one sign, whatever the order of the sum
        if 1e30 < value < 1.1e30:
            x["q"][100] = 1e20                          # +infinity in this row alone; the others give key 7 all their weight
    if name == "do" and np.isfinite(value):
        x["v"] = np.abs(x["v"]) + np.float32(0.5)       # dP of that row overflows to +infinity, its delta too
    x[name][row] = value
    want = visible_f32(x["q"], x["k"], x["v"], x["do"])
    q, k, v, do = (torch.from_numpy(x[n]).cuda()[None, None] for n in ("q", "k", "v", "do"))
    out, lse = tt.attention_forward(q, k, v, causal=True)
    got = (out, lse, *tt.attention_backward(q, k, v, out, lse, do, causal=True))
    tt.check_device_status()
    for what, g, r in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        if what[0] == "d" and 1e30 < value < 1.1e30:
            break                                       # exp(score - lse) of scores near 1e30 is nothing but their rounding
        g = g.cpu().numpy().reshape(r.shape)
        assert np.array_equal(np.isnan(g), np.isnan(r)), what
        assert np.array_equal(np.where(np.isinf(g), np.sign(g), 0), np.where(np.isinf(r), np.sign(r), 0)), what
        ok = np.isfinite(r)
        # two float32 sums of up to 200 terms in different orders; values beyond 1e6 come from the large input: relative to them
        rows = np.abs(np.where(ok, r, 0)).reshape(S, -1).max(1)
        err = np.abs(np.where(ok, g, 0) - np.where(ok, r, 0)).reshape(S, -1).max(1)
        assert bool((err <= 2e-5 * np.maximum(rows, 1.0)).all()), (what, float((err / np.maximum(rows, 1.0)).max()))
