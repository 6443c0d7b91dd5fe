"""Which backward kernels a call takes, at the lines of the choice (both sides of each were timed, see beside the rule)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def single_pass(tt, call):
    tt.capi.profile_enable(True)
    tt.capi.profile_reset()
    try:
        call()
        return "attn_bwd_fused_sm100" in tt.capi.profile_read()
    finally:
        tt.capi.profile_enable(False)
        tt.check_device_status()


@pytest.mark.parametrize("B,H,Hkv,S,L,causal,want", [
    (8, 8, 8, 777, 777, True, True), (4, 32, 32, 300, 300, True, False), (4, 16, 16, 700, 700, False, True), (7, 8, 8, 600, 600, False, False), (16, 32, 32, 128, 128, True, False),
    (1, 40, 40, 100, 4000, False, True), (3, 32, 32, 100, 2000, False, False), (1, 8, 8, 100, 3000, False, True),   # few queries, many keys
    (1, 4, 4, 300, 9000, False, True), (1, 32, 32, 200, 2000, True, True), (2, 8, 8, 3000, 500, False, False), (1, 2, 2, 106, 578, True, False),
    (1, 16, 16, 2048, 2048, False, True), (4, 16, 16, 512, 512, False, False), (1, 8, 8, 3000, 3000, False, False),
    (1, 4, 4, 8192, 8192, True, True), (2, 2, 2, 6900, 6900, True, True), (1, 2, 2, 12288, 12288, True, False), (1, 8, 8, 4096, 4096, True, False), (1, 4, 4, 4096, 4096, True, False)])
def test_dense_head_dim_64(tt, B, H, Hkv, S, L, causal, want):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are in items per SM")
    z = lambda *s: torch.zeros(s, dtype=torch.bfloat16, device="cuda")
    q, k, out, lse = z(B, H, S, 64), z(B, Hkv, L, 64), z(B, H, S, 64), torch.zeros(B, H, S, device="cuda")
    assert single_pass(tt, lambda: tt.attention_backward(q, k, k, out, lse, q, causal=causal)) == want


@pytest.mark.parametrize("n_seq,length,H,Hkv,D,want", [
    (16, 512, 32, 8, 128, False), (16, 768, 32, 8, 128, True), (16, 512, 32, 8, 64, True), (24, 1024, 32, 4, 128, False), (16, 1536, 32, 4, 128, True),
    (24, 512, 32, 32, 128, True), (200, 120, 32, 32, 64, False)])
def test_packed_where_the_single_pass_is_allowed(tt, n_seq, length, H, Hkv, D, want):
    tt.set_backward_deterministic(False)
    n = n_seq * length
    z = lambda h: torch.zeros(n, h, D, dtype=torch.bfloat16, device="cuda")
    cu = torch.arange(0, n + 1, length, dtype=torch.int32, device="cuda")
    q, k, out, lse = z(H), z(Hkv), z(H), torch.zeros(H, n, device="cuda")
    assert single_pass(tt, lambda: tt.attention_backward_varlen(q, k, k, cu, cu, length, length, out, lse, q, causal=True)) == want
