"""Packed backward with workspaces of exactly the size it asks for, between guard bands, by either kernel; and with the size that
the two passes need where the single pass is allowed."""
import ctypes

import pytest

from test_gpu_bwd_packed import packed
from test_gpu_canary import Guarded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def call(tt, q, k, v, do, cu_q, cu_k, mq, mk, causal, ws=None):
    """The backward through the C entry point -> (status, outputs and workspace with their guards, bytes asked for)."""
    out, lse = tt.attention_forward_varlen(q, k, v, cu_q, cu_k, mq, mk, causal=causal)
    d = tt.capi.VarlenDesc(n_seq=len(cu_q) - 1, H=q.shape[1], Hkv=k.shape[1], D=q.shape[2], dtype=tt.capi.TT_BF16, causal=int(causal),
                           max_q=mq, max_k=mk, total_q=q.shape[0], total_k=k.shape[0])
    lib = tt.capi.lib
    need = int(lib.tt_attn_bwd_varlen_workspace_bytes(ctypes.byref(d)))
    g = [Guarded(t.shape, torch.bfloat16) for t in (q, k, v)] + [Guarded((need if ws is None else ws,), torch.uint8)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.tt_attn_bwd_varlen(ctypes.byref(d), p(q), p(k), p(v), p(cu_q), p(cu_k), p(out), p(lse), p(do), *(p(x.t) for x in g),
                                ctypes.c_size_t(g[3].n), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    tt.check_device_status()
    return rc, g, need


@pytest.mark.parametrize("path", ["two_pass", "fused"])
@pytest.mark.parametrize("lens_q,lens_k,H,Hkv,D,lead,tail,causal", [
    ([1, 127, 128, 129, 256, 257], None, 2, 2, 128, 0, 0, True), ([0, 300, 0, 131, 0], None, 4, 2, 64, 5, 130, False),
    ([200, 1, 0, 140], [90, 400, 77, 0], 2, 1, 128, 129, 1, True), ([1] * 40, None, 3, 3, 64, 0, 0, True)])
def test_guards_and_tokens_of_no_sequence(tt, monkeypatch, path, lens_q, lens_k, H, Hkv, D, lead, tail, causal):
    monkeypatch.setenv("TT_BWD_PATH", path)
    q, k, v, do, *rest = packed(lens_q, lens_k or lens_q, H, Hkv, D, lead, tail, 11)
    rc, g, _ = call(tt, q, k, v, do, *rest, causal)
    assert rc == 0
    for name, x in zip(("dq", "dk", "dv", "workspace"), g):
        assert x.intact(), f"{name}: a guard band was written"
    for x in g[:3]:
        assert not x.t[:lead].any() and not x.t[x.t.shape[0] - tail:].any() and torch.isfinite(x.t.float()).all()


def test_a_small_workspace_takes_the_two_passes(tt):
    n = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    args = packed([128] * n, [128] * n, 1, 1, 128, 0, 0, 1)
    tt.set_backward_deterministic(True)
    try:
        rc, want, small = call(tt, *args, True)
    finally:
        tt.set_backward_deterministic(False)
    rc2, got, large = call(tt, *args, True, ws=small)
    assert rc == rc2 == 0 and large > small
    assert all(torch.equal(a.t, b.t) and b.intact() for a, b in zip(want[:3], got[:3])) and got[3].intact()
    assert call(tt, *args, True, ws=small - 256)[0] == tt.capi.TT_ERR_WORKSPACE
