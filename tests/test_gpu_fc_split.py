"""The fully connected layer where its kernels cut K among the CTAs of a cluster (fc_gemm_sm100.cu), against float64.

Bounds.  bf16: inputs are exact, sums are float32, the result is rounded once: 2^-8 of the value plus the sums' rounding, below
2^-20 of the row's sum of magnitudes."""
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
