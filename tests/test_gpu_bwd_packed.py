"""The single-pass backward on packed batches against the two passes on the same inputs, and the choice between them."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def packed(lens_q, lens_k, H, Hkv, D, lead, tail, seed):
    """Sequences behind `lead` tokens of no sequence and before `tail` more."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda rows, h: torch.randn(rows, h, D, generator=g, device="cuda").bfloat16()
    cu = lambda lens: torch.tensor([lead + sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
    tq, tk = lead + sum(lens_q) + tail, lead + sum(lens_k) + tail
    return n(tq, H) * 0.5, n(tk, Hkv) * 0.5, n(tk, Hkv) * 0.5, n(tq, H), cu(lens_q), cu(lens_k), max(max(lens_q), 1), max(max(lens_k), 1)


MANY = [(37 * i) % 300 for i in range(70)]     # more sequences than a warp has lanes: the search takes two steps
CASES = [   # lengths around the tile, one tile more or less after the numbering's rounding, empty sequences on either side
    ([128], [128], 1, 1, 128, 0, 0, True),
    ([1, 127, 128, 129, 256, 257], None, 2, 2, 128, 0, 0, True),
    ([1, 127, 128, 129, 256, 257], None, 4, 2, 64, 5, 130, False),
    ([0, 300, 0, 0, 131, 0], None, 2, 1, 128, 3, 1, True),
    ([200, 1, 0, 140], [90, 400, 77, 0], 4, 1, 128, 0, 7, True),     # fewer keys than queries, and more
    ([200, 1, 0, 140], [90, 400, 77, 0], 2, 2, 64, 129, 0, False),
    (MANY, None, 3, 3, 64, 1, 2, True),
    (MANY, MANY[::-1], 2, 2, 128, 0, 300, False),
    ([700] * 9, None, 16, 16, 128, 0, 0, True),                      # several items per SM
]


@pytest.mark.parametrize("lens_q,lens_k,H,Hkv,D,lead,tail,causal", CASES)
def test_single_pass_equals_two_passes(tt, monkeypatch, lens_q, lens_k, H, Hkv, D, lead, tail, causal):
    lens_k = lens_k or lens_q
    q, k, v, do, cu_q, cu_k, mq, mk = packed(lens_q, lens_k, H, Hkv, D, lead, tail, len(lens_q) + D)
    out, lse = tt.attention_forward_varlen(q, k, v, cu_q, cu_k, mq, mk, causal=causal)
    got = {}
    for path in ("two_pass", "fused"):
        monkeypatch.setenv("TT_BWD_PATH", path)
        bad = [torch.full_like(t, float("nan")) for t in (q, k, v)]     # what the allocator hands out next is not zero
        del bad
        got[path] = tt.attention_backward_varlen(q, k, v, cu_q, cu_k, mq, mk, out, lse, do, causal=causal)
        tt.check_device_status()
    # the same products and float sums in another order, one rounding to bf16 each: within one step of bf16 at the tensor's
    # size (dK and dV sums differ in nothing but the order, dQ's tiles are added as they come)
    for name, a, b in zip(("dq", "dk", "dv"), got["fused"], got["two_pass"]):
        assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * max(float(b.float().abs().max()), 1e-3), name
    for t in got["fused"]:
        assert not t[:lead].any() and not t[t.shape[0] - tail:].any()


def test_choice_by_items_per_sm(tt):
    """Three key tiles per SM: the two passes below, the single pass from there on, the two passes again where results must repeat."""
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count

    def names(tiles, deterministic=False):
        q, k, v, do, cu, _, m, _ = packed([128] * tiles, [128] * tiles, 1, 1, 128, 0, 0, 1)
        out, lse = tt.attention_forward_varlen(q, k, v, cu, cu, m, m)
        tt.set_backward_deterministic(deterministic)
        tt.capi.profile_enable(True)
        tt.capi.profile_reset()
        try:
            tt.attention_backward_varlen(q, k, v, cu, cu, m, m, out, lse, do)
            return set(tt.capi.profile_read())
        finally:
            tt.capi.profile_enable(False)
            tt.set_backward_deterministic(False)
    assert "attn_bwd_fused_sm100" not in names(3 * n_sm - 1)
    assert "attn_bwd_fused_sm100" in names(3 * n_sm)
    assert "attn_bwd_fused_sm100" not in names(3 * n_sm, deterministic=True)
    tt.check_device_status()
