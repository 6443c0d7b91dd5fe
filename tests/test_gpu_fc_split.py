"""The fully connected layer where its kernels cut K among the CTAs of a cluster (fc_gemm_sm100.cu, fc_f32_sm100.cu), and float
tensors on the tensor cores as three bf16 parts, against float64.

Bounds.  bf16: inputs are exact, sums are float32, the result is rounded once: 2^-8 of the value plus the sums' rounding, below
2^-20 of the row's sum of magnitudes.  Float: a product loses below 2^-23 to the terms left out, a chunk of 64 a few units of
2^-23 to truncating additions, chunks are added in float32: 2^-20 of the sum of magnitudes covers it (K up to 64 chunks)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(tt, x, w, b, dy, slack):
    y = tt.fc_forward(x, w, b)
    dx, dw, db = tt.fc_backward(x, w, dy)
    tt.check_device_status()
    x6, w6, b6, dy6 = (t.double() for t in (x, w, b, dy))
    for name, got, want, mags in (("y", y, x6 @ w6 + b6, x6.abs() @ w6.abs() + b6.abs()), ("dx", dx, dy6 @ w6.t(), dy6.abs() @ w6.abs().t()),
                                  ("dw", dw, x6.t() @ dy6, x6.abs().t() @ dy6.abs()), ("db", db, dy6.sum(0), dy6.abs().sum(0))):
        assert got.shape == want.shape
        bound = 2.0 ** -20 * mags + slack * want.abs()
        assert bool(((got.double() - want).abs() <= bound).all()), (name, float(((got.double() - want).abs() / bound).max()))


# one tile over long K in each direction, shares of unequal length (33 blocks of 64 over 8 CTAs: the last has fewer, 9 over 2),
# remainders of a block, tile edges in M and N
@pytest.mark.parametrize("rows,fin,fout", [(2112, 64, 40), (32, 8192, 16), (100, 72, 8192), (577, 576, 264), (130, 2056, 520), (16384, 8, 8)])
def test_bf16_cut_along_k(tt, rows, fin, fout):
    g = torch.Generator(device="cuda").manual_seed(rows + fin)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    check(tt, n(rows, fin), n(fin, fout), n(fout), n(rows, fout), 2.0 ** -8)


# pitches that are and are not multiples of 4 and 8, tile and chunk edges, one CTA per tile and clusters
@pytest.mark.parametrize("rows,fin,fout", [(128, 128, 128), (129, 65, 127), (640, 333, 130), (64, 1000, 36), (33, 4095, 11), (4099, 129, 260),
                                           (1500, 1500, 1028), (1, 3, 1)])
def test_float_parts(tt, rows, fin, fout):
    g = torch.Generator(device="cuda").manual_seed(rows + fin)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda")
    check(tt, n(rows, fin), n(fin, fout), n(fout), n(rows, fout), 2.0 ** -23)


def test_float_pointers_off_16_bytes(tt):
    g = torch.Generator(device="cuda").manual_seed(1)
    n = lambda r, c: torch.randn(r * c + 1, generator=g, device="cuda")[1:].view(r, c)
    check(tt, n(200, 256), n(256, 132), torch.randn(132, generator=g, device="cuda"), n(200, 132), 2.0 ** -23)


def test_float_extremes(tt):
    """The largest finite float keeps its value; infinities and NaN give what plain additions and multiplications give, in
    their rows and columns only."""
    x = torch.ones(300, 200, device="cuda")
    w = torch.full((200, 140), 2.0 ** -10, device="cuda")
    big = torch.finfo(torch.float32).max
    x[3, 5], x[4, 6] = big, -big
    y = tt.fc_forward(x, w)
    assert torch.allclose(y.double(), x.double() @ w.double(), rtol=1e-6, atol=0)
    x[150, 7], x[151, 8], x[152, 9] = float("inf"), float("-inf"), float("nan")
    w[0, 139] = float("inf")
    y = tt.fc_forward(x, w)
    tt.check_device_status()
    want = x.double() @ w.double()
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert torch.equal(torch.isinf(y)[ok], torch.isinf(want)[ok]) and torch.equal(torch.sign(y)[ok].double(), torch.sign(want)[ok])
    fin = torch.isfinite(want)
    assert torch.allclose(y.double()[fin], want[fin], rtol=1e-6, atol=0)


@pytest.mark.parametrize("fin", [64, 1000, 8192])   # one CTA per tile, and clusters that cut K
def test_float_products_that_overflow(tt, fin):
    """Finite factors whose product overflows give the infinity of the product's sign, whatever the signs of their parts'
    remainders (1.0039 rounds up to its first part, 1.0009 down), forward and in both gradients; products that just fit stay finite."""
    x, w = torch.ones(150, fin, device="cuda"), torch.ones(fin, 136, device="cuda")
    x[0], x[1], x[2], x[140] = 1.0039e30, -4 * 1.0039e30, 16 * 1.0009e30, -64 * 1.0009e30   # (sums that do not cancel)
    w[:, 3], w[:, 135] = 1e20, -4e20
    x[5, 7], w[7, 9] = 1.8e19, 1.8e19            # 3.24e38: finite
    dy = torch.ones(150, 136, device="cuda")
    dy[0, 3] = 1.0039e20                         # dx[0] = dy w^T and dw[:, 3] = x^T dy overflow
    y = tt.fc_forward(x, w)
    dx, dw, _ = tt.fc_backward(x, w, dy)
    tt.check_device_status()
    for name, got, want in (("y", y, x.double() @ w.double()), ("dx", dx, dy.double() @ w.double().t()), ("dw", dw, x.double().t() @ dy.double())):
        over = want.abs() > torch.finfo(torch.float32).max
        assert bool((got[over] == want[over].sign().float() * float("inf")).all()), name
        assert torch.allclose(got[~over].double(), want[~over], rtol=1e-5, atol=0), name
    assert bool(torch.isinf(y).any()) and bool(torch.isinf(dx).any()) and bool(torch.isinf(dw).any())


def test_float_rows_up_to_the_last_32_bit_number(tt):
    """2^31 - 1 rows: tiles and row numbers end at the largest int."""
    rows = 2 ** 31 - 1
    x = torch.full((rows, 1), 3.0, device="cuda")
    x[-1], x[-130], x[0] = 5.0, 7.0, 11.0
    y = tt.fc_forward(x, torch.full((1, 1), 2.0, device="cuda"))
    tt.check_device_status()
    for a, b in zip(y.split(1 << 28), x.split(1 << 28)):
        assert torch.equal(a, 2.0 * b)
