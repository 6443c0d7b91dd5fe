"""A device-side wait that has given up ends its own launch early and no other: calls made before the host has looked at the
status word compute everything."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def expire(tt):
    tt.capi.check(tt.capi.lib.tt_debug_wait_timeout(2_000_000, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


def poison(*like):
    """Leaves the freed blocks that outputs of these shapes take next full of sevens."""
    held = [torch.full_like(t, 7.0) for t in like for _ in range(2)]
    del held


# more items than SMs in every launch, so that some CTAs start late
@pytest.mark.parametrize("dtype,D,group", [(torch.float32, 64, 1), (torch.float32, 128, 2), (torch.bfloat16, 64, 1), (torch.bfloat16, 128, 1),
                                           (torch.bfloat16, 128, 4)])
def test_calls_after_an_expired_wait_are_complete(tt, dtype, D, group):
    g = torch.Generator(device="cuda").manual_seed(D)
    n = lambda h: torch.randn(4, h, 300, D, generator=g, device="cuda").to(dtype)
    q, do, k, v = n(64), n(64), n(64 // group), n(64 // group)
    want = tt.attention_forward(q, k, v, causal=True)
    want += tt.attention_backward(q, k, v, *want, do, causal=True)
    tt.check_device_status()
    expire(tt)
    poison(*want)
    got = tt.attention_forward(q, k, v, causal=True)
    got += tt.attention_backward(q, k, v, *got, do, causal=True)
    with pytest.raises(tt.TTError) as err:   # still reported, as what it was
        tt.check_device_status()
    assert err.value.code == tt.capi.TT_ERR_TIMEOUT and "barrier id 99" in str(err.value)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), want, got):
        if name == "dq" and dtype == torch.bfloat16 and D == 64:   # added up in any order: the last bit of a bf16 value
            assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * float(a.float().abs().max())
        else:
            assert torch.equal(a, b), name


def test_packed_batch_after_an_expired_wait_is_complete(tt):
    g = torch.Generator(device="cuda").manual_seed(1)
    cu = torch.tensor([0, 300, 301, 900, 1600], dtype=torch.int32, device="cuda")
    q, k, v, do = (torch.randn(1600, 32, 128, generator=g, device="cuda").bfloat16() for _ in range(4))
    want = tt.attention_forward_varlen(q, k, v, cu, cu, 700, 700, causal=True)
    want += tt.attention_backward_varlen(q, k, v, cu, cu, 700, 700, *want, do, causal=True)
    tt.check_device_status()
    expire(tt)
    poison(*want)
    got = tt.attention_forward_varlen(q, k, v, cu, cu, 700, 700, causal=True)
    got += tt.attention_backward_varlen(q, k, v, cu, cu, 700, 700, *got, do, causal=True)
    with pytest.raises(tt.TTError):
        tt.check_device_status()
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), want, got):
        assert torch.equal(a, b), name


def test_a_cta_that_gave_up_drops_the_rest_of_its_launch(tt):
    """20000 one-warp CTAs (at most 32 run on an SM) wait for about 5 ms each.  Those of the first wave give up and cancel the
    others; the launch behind them is untouched."""
    fn = tt.capi.lib.tt_debug_wait_timeout_grid
    fn.restype, fn.argtypes = ctypes.c_int, [ctypes.c_int64, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    started = torch.zeros(2, dtype=torch.int32, device="cuda")
    tt.check_device_status()
    tt.capi.check(fn(10_000_000, 20000, ctypes.c_void_p(started.data_ptr()), st))
    tt.capi.check(fn(2_000_000, 7, ctypes.c_void_p(started.data_ptr() + 4), st))
    with pytest.raises(tt.TTError) as err:
        tt.check_device_status()
    assert err.value.code == tt.capi.TT_ERR_TIMEOUT
    first, second = started.tolist()
    resident = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    # dropping starts with the first CTA that gives up; until the last one has been dropped, a few take the places that become free
    assert 1 <= first < 2 * resident and second == 7, (first, second)
