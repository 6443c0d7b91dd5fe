"""Size of the backward's workspace: of a packed batch a function of the token count, however many sequences share it."""
import ctypes

import pytest


def varlen_bytes(tt, n_seq, total, H, D, longest):
    d = tt.capi.VarlenDesc(n_seq=n_seq, H=H, D=D, dtype=tt.capi.TT_BF16, causal=1, max_q=longest, max_k=longest, total_q=total, total_k=total)
    return int(tt.capi.lib.tt_attn_bwd_varlen_workspace_bytes(ctypes.byref(d)))


def two_pass_bytes(total, H):
    return 2 * ((total * H * 4 + 255) // 256 * 256)


# many sequences of one token up, the last two long enough for the single pass
BATCHES = [(10000, 20, 32, 128), (4096, 64, 32, 128), (50000, 1, 8, 64), (100, 127, 32, 128), (16, 2048, 32, 128), (444, 128, 1, 128)]


@pytest.mark.parametrize("n_seq,length,H,D", BATCHES)
def test_two_passes_need_their_statistics_alone(tt, n_seq, length, H, D):
    tt.set_backward_deterministic(True)
    try:
        assert varlen_bytes(tt, n_seq, n_seq * length, H, D, length) == two_pass_bytes(n_seq * length, H)
    finally:
        tt.set_backward_deterministic(False)


@pytest.mark.parametrize("n_seq,length,H,D", BATCHES)
def test_single_pass_takes_no_more_than_twice_its_rows(tt, n_seq, length, H, D):
    tt.set_backward_deterministic(False)
    got, rows = varlen_bytes(tt, n_seq, n_seq * length, H, D, length), n_seq * length * H
    assert got <= max(two_pass_bytes(n_seq * length, H), 2 * rows * (D + 2) * 4)
    if length >= 128:
        assert got >= rows * (D + 2) * 4


@pytest.mark.parametrize("B,H,S,D", [(1, 64, 32768, 128), (4, 32, 4096, 128), (8, 16, 1024, 64), (2, 3, 300, 64)])
def test_dense_calls_need_one_accumulator_and_one_pair_of_statistics(tt, B, H, S, D):
    d = tt.capi.make_desc(B, H, S, S, D, tt.capi.TT_BF16, True, None)
    assert int(tt.capi.lib.tt_attn_bwd_workspace_bytes(ctypes.byref(d))) == B * H * (-(-S // 128) * 128) * (D + 2) * 4
