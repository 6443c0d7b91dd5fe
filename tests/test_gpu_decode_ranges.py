"""Decode whose keys are cut into ranges of whole 128-key tiles: key counts that nothing divides, few slices (one wave of ranges), slices
that would leave a last wave nearly empty, ragged lengths whose later ranges are empty.  Against the oracle, out 2e-2 absolute and
log-sum-exp 1e-3 as for the base op; partial results are floats, so the ranges add no rounding of their own."""
import numpy as np
import pytest

from test_gpu_variants import dense_decode_ref, make_grouped

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def run(tt, oracle, B, H, Hkv, L, D, lens=None):
    q, k, v, _ = make_grouped(oracle, L + D, B, H, Hkv, 1, L, D, True)
    o_r, lse_r = dense_decode_ref(oracle, q, k, v) if lens is None else dense_decode_ref(oracle, q, k, v, np.asarray(lens, np.int32))
    tq, tk, tv = (torch.from_numpy(a).cuda().bfloat16() for a in (q, k, v))
    before = tt.capi.launch_count()
    if lens is None:
        out, lse = tt.attention_decode(tq, tk, tv)
    else:
        out, lse = tt.attention_decode_paged(tq, tk, tv, seq_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"))
    launches = tt.capi.launch_count() - before
    tt.check_device_status()
    assert oracle.max_abs_err(out.float().cpu().numpy(), o_r) <= 2e-2
    got = lse.cpu().numpy()
    keep = np.isfinite(lse_r)
    assert np.array_equal(np.isfinite(got), keep) and oracle.max_abs_err(got[keep], lse_r[keep]) <= 1e-3
    return launches


# the last: one slice cut into as many ranges as the rule for groups up to 16 gives, 128
@pytest.mark.parametrize("B,H,Hkv,L,D", [(1, 4, 4, 1024, 64), (1, 8, 2, 1025, 128), (1, 32, 8, 5003, 128), (1, 16, 1, 16385, 128),
                                          (38, 8, 8, 2051, 64), (1, 2, 1, 66001, 64)])
def test_dense_ranges(tt, oracle, B, H, Hkv, L, D):
    assert run(tt, oracle, B, H, Hkv, L, D) == 2


def test_short_cache_is_one_launch(tt, oracle):
    assert run(tt, oracle, 2, 8, 2, 1023, 128) == 1


@pytest.mark.parametrize("H,Hkv,D", [(8, 2, 128), (4, 4, 64)])
def test_ragged_ranges_with_empty_ones(tt, oracle, H, Hkv, D):
    lens = [0, 1, 1024, 1025, 2048, 2300, 127, 128] * 5
    assert run(tt, oracle, len(lens), H, Hkv, 2300, D, lens) == 2


# Groups above 16 run on the forward kernel, whose rules give up to two ranges per SM: here (148 SMs) 144, 256, 147 and 129.
@pytest.mark.parametrize("H,Hkv,L,D,page", [(32, 1, 36864, 128, 0), (32, 1, 65536, 64, 0), (64, 2, 131072, 64, 128), (32, 1, 33024, 128, 64)])
def test_more_ranges_than_the_merge_holds_in_registers(tt, oracle, H, Hkv, L, D, page):
    G = H // Hkv
    q, k, v, _ = oracle.make_inputs(L + D, 1, Hkv, G, L, D)   # a group's heads as query rows
    q, k, v = (oracle.bf16_round(a) for a in (q, k, v))
    o_r, lse_r = oracle.attention_forward(q, k, v, False)
    tq = torch.from_numpy(q).cuda().bfloat16().view(1, H, 1, D)
    tk, tv = (torch.from_numpy(a).cuda().bfloat16() for a in (k, v))
    before = tt.capi.launch_count()
    if page:
        n = L // page
        order = torch.randperm(n, generator=torch.Generator().manual_seed(L))
        pool = lambda t: t[0].view(Hkv, n, page, D).transpose(0, 1)[torch.argsort(order).cuda()].contiguous()   # page i of the cache at order[i]
        out, lse = tt.attention_decode_paged(tq, pool(tk), pool(tv), block_table=order.to(torch.int32).cuda().view(1, n))
    else:
        out, lse = tt.attention_decode(tq, tk, tv)
    assert tt.capi.launch_count() - before == 2
    tt.check_device_status()
    # 2-norm, because sums over this many keys are far below 2e-2: the probabilities, a range's result and the output are each
    # rounded to bf16, by 2^-9 of themselves at most
    got = out.float().cpu().numpy().reshape(o_r.shape)
    assert float(np.linalg.norm(got - o_r)) <= 3 * 2.0 ** -9 * float(np.linalg.norm(o_r))
    assert oracle.max_abs_err(lse.cpu().numpy().reshape(lse_r.shape), lse_r) <= 1e-3
