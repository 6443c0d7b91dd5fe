"""Both packed backwards against the float32 oracle, sequence by sequence and head by head, so that an error in one short sequence is not
hidden by the gradients of another; and the single pass against the two passes in the same way."""
import numpy as np
import pytest

import test_gpu_varlen as varlen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def spread(n, lo, hi):
    return [lo + (i * 7919) % (hi - lo + 1) for i in range(n)]


def slices(lens, heads):
    at = 0
    for n in lens:
        for h in range(heads):
            if n:
                yield slice(at, at + n), h
        at += n


# beside those cases: above three key tiles per SM, where a caller who allows it gets the single pass, and more sequences than two steps of the
# search find
CASES = varlen.CASES + [(spread(14, 300, 900), None, 8, 8, 128, True), (spread(9, 200, 1100), spread(9, 600, 900), 16, 8, 64, False),
                        ([i % 4 for i in range(1100)], None, 2, 1, 64, True)]


@pytest.mark.parametrize("path", ["fused", "two_pass"])
@pytest.mark.parametrize("lens_q,lens_k,H,Hkv,D,causal", CASES)
def test_every_sequence_and_head(tt, oracle, monkeypatch, path, lens_q, lens_k, H, Hkv, D, causal):
    monkeypatch.setenv("TT_BWD_PATH", path)
    lens_k = lens_q if lens_k is None else lens_k
    q, k, v, do = varlen._pack(oracle, 5 + H + D, lens_q, lens_k, H, Hkv, D)
    _, _, *want = varlen._oracle_packed(oracle, q, k, v, do, lens_q, lens_k, causal)
    dev = lambda x: torch.from_numpy(x).to("cuda", dtype=torch.bfloat16)
    cu = lambda lens: torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    args = (dev(q), dev(k), dev(v), cu(lens_q), cu(lens_k), max(lens_q), max(lens_k))
    out, lse = tt.attention_forward_varlen(*args, causal=causal)
    got = [t.float().cpu().numpy() for t in tt.attention_backward_varlen(*args, out, lse, dev(do), causal=causal)]
    tt.check_device_status()
    for name, g, w, lens, heads in zip(("dq", "dk", "dv"), got, want, (lens_q, lens_k, lens_k), (H, Hkv, Hkv)):
        for s, h in slices(lens, heads):
            assert oracle.max_abs_err(g[s, h], w[s, h]) <= oracle.bf16_grad_tol(w[s, h]), (name, s, h)


@pytest.mark.parametrize("B,H,Hkv,S,L,D,causal", [(1, 2, 2, 384, 384, 64, True), (1, 1, 1, 300, 300, 128, True), (1, 2, 2, 130, 515, 64, True),
                                                  (2, 4, 2, 1024, 1024, 128, True), (1, 1, 1, 257, 129, 128, False)])
def test_dense_single_pass_within_one_step_of_the_two_passes(tt, monkeypatch, B, H, Hkv, S, L, D, causal):
    """Both form dS from the float P and sum in float: what differs is the order of the sums, at most one step of bf16 at a slice's size."""
    g = torch.Generator(device="cuda").manual_seed(S)
    n = lambda h, s: torch.randn(B, h, s, D, generator=g, device="cuda").bfloat16()
    q, k, v, do = n(H, S) * 0.5, n(Hkv, L) * 0.5, n(Hkv, L), n(H, S)
    out, lse = tt.attention_forward(q, k, v, causal=causal)
    got = {}
    for path in ("fused", "two_pass"):
        monkeypatch.setenv("TT_BWD_PATH", path)
        got[path] = tt.attention_backward(q, k, v, out, lse, do, causal=causal)
    tt.check_device_status()
    for name, a, b in zip(("dq", "dk", "dv"), got["fused"], got["two_pass"]):
        far, size = (a.float() - b.float()).abs().amax((2, 3)), b.float().abs().amax((2, 3))
        assert bool((far <= 2.0 ** -7 * size).all()), name
