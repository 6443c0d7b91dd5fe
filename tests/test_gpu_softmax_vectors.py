"""Row softmax at pitches off the 16-byte vectors, at every change of the threads that hold a row (4 to 32 lanes, a CTA, a CTA that
reads it twice), and from pointers off 16 bytes, against float64.

Bounds.  Forward, float: the exponential's argument is rounded to 2^-24 of at most 32, and __expf adds about as much again: 2^-18 of the
value; bf16 rounds the result once more, 2^-8.  Backward: sum(y dy) is a float32 sum of values whose magnitudes add to at most
max|dy|, so y (2^-19 max|dy|) beside the rounding of the result."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def placed(flat_values, rows, cols, offset):
    """[rows, cols] inside a larger buffer whose other values must not change."""
    buf = torch.full((rows * cols + 64,), 777.0, device="cuda", dtype=flat_values.dtype)
    view = buf[32 + offset:32 + offset + rows * cols].view(rows, cols)
    view.copy_(flat_values.view(rows, cols))
    return buf, view


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_every_row_length(tt, dtype, offset):
    cols_list = [1, 3, 5, 7, 8, 9, 15, 16, 17, 31, 33, 63, 65, 127, 129, 255, 257, 511, 513, 1023, 1025, 2047, 2049, 2056, 4095, 4097, 8191,
                 8193, 16383, 16385, 24001, 32769, 65535, 131072, 131073]
    slack = 2.0 ** -18 if dtype is torch.float32 else 2.0 ** -8
    for cols in cols_list:
        rows = 37 if cols < 5000 else 3
        g = torch.Generator(device="cuda").manual_seed(cols)
        _, x = placed(torch.randn(rows * cols, generator=g, device="cuda").mul_(3).to(dtype), rows, cols, offset)
        _, dy = placed(torch.randn(rows * cols, generator=g, device="cuda").to(dtype), rows, cols, offset)
        buf, y = placed(torch.zeros(rows * cols, device="cuda", dtype=dtype), rows, cols, offset)
        tt.softmax_forward(x, out=y)
        want = torch.softmax(x.double(), -1)
        assert bool(((y.double() - want).abs() <= slack * want + 1e-38).all()), cols
        dx = tt.softmax_backward(y, dy)
        y6, d6 = y.double(), dy.double()
        want = y6 * (d6 - (y6 * d6).sum(-1, keepdim=True))
        assert bool(((dx.double() - want).abs() <= slack * want.abs() + y6 * d6.abs().max() * 2.0 ** -19 + 1e-38).all()), cols
        tt.softmax_forward(x, out=x)                      # in place: neighbouring rows share vectors
        assert torch.equal(x, y), cols
        n = rows * cols
        assert bool((buf[:32 + offset] == 777).all()) and bool((buf[32 + offset + n:] == 777).all()), cols


@pytest.mark.parametrize("cols", [13, 1023, 3001, 40001])
def test_masked_and_infinite_rows(tt, cols):
    """The type's lowest value and -inf as masks, a row of them, an infinity and a NaN: as plain exp and sums give them."""
    x = torch.randn(6, cols, device="cuda")
    x[0, ::2] = torch.finfo(torch.float32).min
    x[1, 1::2] = float("-inf")
    x[2] = torch.finfo(torch.float32).min
    x[3] = float("-inf")
    x[4, cols // 2] = float("inf")
    x[5, cols - 1] = float("nan")
    y, want = tt.softmax_forward(x).double(), torch.softmax(x.double(), -1)
    assert torch.allclose(y[:3], want[:3], rtol=2.0 ** -18, atol=1e-38)
    assert bool(torch.isnan(y[3]).all()) and bool(torch.isnan(y[5]).all()) and bool(torch.isnan(y[4, cols // 2]))
