"""Arguments of the torch calls: lengths and scales are whatever int() and float() take, and no length is cut to 32 bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_lengths_and_scale_of_any_number_type(tt):
    q = torch.randn(300, 4, 64, device="cuda").bfloat16()
    cu = torch.tensor([0, 100, 300], dtype=torch.int32, device="cuda")
    want = tt.attention_forward_varlen(q, q, q, cu, cu, 200, 200, scale=0.25)
    for n, scale in ((200.0, np.float32(0.25)), (np.int64(200), torch.tensor(0.25)), (torch.tensor(200), "0.25"), ("200", 0.25)):
        got = tt.attention_forward_varlen(q, q, q, cu, cu, n, n, scale=scale)
        assert all(torch.equal(a, b) for a, b in zip(want, got))
        grads = tt.attention_backward_varlen(q, q, q, cu, cu, n, n, *got, q, scale=scale)
        assert all(g.shape == q.shape for g in grads)
    k = torch.randn(2, 4, 500, 64, device="cuda").bfloat16()
    one = torch.randn(2, 8, 1, 64, device="cuda").bfloat16()
    want = tt.attention_decode_paged(one, k, k, max_len=400)
    for n in (400.0, np.int32(400), torch.tensor(400.0)):
        assert all(torch.equal(a, b) for a, b in zip(want, tt.attention_decode_paged(one, k, k, max_len=n)))
    with pytest.raises(TypeError):
        tt.attention_decode_paged(one, k, k, max_len=[400])


def test_lengths_beyond_32_bits_are_refused(tt):
    k = torch.randn(2, 4, 500, 64, device="cuda").bfloat16()
    one = torch.randn(2, 8, 1, 64, device="cuda").bfloat16()
    for n in (501, 2 ** 32 + 400, 2 ** 33):
        with pytest.raises(ValueError):
            tt.attention_decode_paged(one, k, k, max_len=n)
    q = torch.randn(300, 4, 64, device="cuda").bfloat16()
    cu = torch.tensor([0, 100, 300], dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError):
        tt.attention_forward_varlen(q, q, q, cu, cu, 2 ** 32 + 200, 200)
