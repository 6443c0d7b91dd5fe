"""Order and numbering of the packed forward's work items: up to 32 sequences (the loader holds their lengths) and more (it
searches), one phase and two, against the float32 oracle and, where the oracle would take too long, against the dense call."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def batch(lens, H, Hkv, D, lead, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lead + sum(lens)
    cu = torch.tensor([lead + sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
    r = lambda h: (torch.randn(n, h, D, generator=g, device="cuda") * 0.6).bfloat16()
    return r(H), r(Hkv), r(Hkv), cu


def spread(n, lo, hi):
    return [lo + (i * 7919) % (hi - lo + 1) for i in range(n)]


CASES = [   # lengths, heads, key/value heads, D, tokens of no sequence ahead, causal
    ([1100, 0, 257, 0, 0, 900, 256, 1], 2, 1, 128, 0, True),             # empty sequences between the light blocks, and at neither end
    ([0, 0, 1500, 300, 0], 1, 1, 64, 700, True),                         # ... and at both, behind tokens of none
    ([2048], 2, 2, 128, 300, True),
    (spread(31, 0, 1400), 1, 1, 64, 5, True),                            # a lane short of the registers' number, as many, one more
    (spread(32, 0, 1400), 1, 1, 128, 0, True),
    (spread(33, 0, 1400), 1, 1, 64, 0, True),
    (spread(32, 0, 300), 2, 2, 128, 130, False),
    (spread(70, 0, 1300), 2, 2, 128, 3, False),
    ([1 + i % 3 for i in range(1100)], 1, 1, 64, 0, True),               # the search takes three steps
]


@pytest.mark.parametrize("lens,H,Hkv,D,lead,causal", CASES)
def test_packed_forward_against_the_oracle(tt, oracle, lens, H, Hkv, D, lead, causal):
    q, k, v, cu = batch(lens, H, Hkv, D, lead, len(lens))
    out, lse = tt.attention_forward_varlen(q, k, v, cu, cu, max(lens), max(lens), causal=causal)
    tt.check_device_status()
    f = lambda t: t.permute(1, 0, 2)[None].float().cpu().numpy()
    at = lead
    for n in lens:
        if n:
            s = slice(at, at + n)
            want, want_lse = oracle.attention_forward(f(q[s]), oracle.expand_kv_heads(f(k[s]), H), oracle.expand_kv_heads(f(v[s]), H), causal)
            assert oracle.max_abs_err(f(out[s]), want) <= 2e-2
            assert oracle.max_abs_err(lse[:, s][None].cpu().numpy(), want_lse) <= 2e-2
        at += n


@pytest.mark.parametrize("n_seq,H,D", [(9, 24, 128), (9, 24, 64), (40, 24, 128), (40, 24, 64), (36, 4, 64)])
def test_many_items_per_sm_equal_the_dense_call(tt, n_seq, H, D):
    """Causal, with light blocks, above and below the numbers of items per SM where the order changes."""
    S = 1100
    q, k, v, cu = batch([S] * n_seq, H, H, D, 0, n_seq)
    out, lse = tt.attention_forward_varlen(q, k, v, cu, cu, S, S, causal=True)
    dense = lambda t: t.reshape(n_seq, S, H, D).permute(0, 2, 1, 3).contiguous()
    want, want_lse = tt.attention_forward(dense(q), dense(k), dense(v), causal=True)
    tt.check_device_status()
    assert torch.equal(dense(out), want)
    assert torch.equal(lse.reshape(H, n_seq, S).permute(1, 0, 2), want_lse)
