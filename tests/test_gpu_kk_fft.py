"""The FFT Kramers-Kronig transform (kk_fft.cu) against 80-bit direct sums: grid
lengths around powers of two, the largest one and the direct kernel beyond it, zero,
mixed-scale and non-finite rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kk_longdouble(re, im):
    """re + (2/pi) sum K im, im + (2/pi) sum K re with K_fs = s / (s^2 - f^2), s != f."""
    n = re.shape[1]
    s = np.arange(n, dtype=np.longdouble)
    with np.errstate(divide="ignore", invalid="ignore"):
        K = s[None, :] / ((s[None, :] - s[:, None]) * (s[None, :] + s[:, None]))
    np.fill_diagonal(K, 0.0)
    c = np.longdouble(2) / (4 * np.arctan(np.longdouble(1)))
    a, b = re.astype(np.longdouble), im.astype(np.longdouble)
    return a + c * (b @ K.T), b + c * (a @ K.T)


# the sums have nf terms of up to |x|; 2 nf eps covers both a direct sum and the
# transform, log2(L) eps times the row's norm
@pytest.mark.parametrize("nf", [1, 2, 3, 8, 9, 17, 31, 64, 65, 128, 129, 257, 511, 1000, 1025, 2000, 2049, 4096, 4097])
def test_kk_fft_vs_longdouble(ctx, nf):
    rng = np.random.default_rng(nf)
    rows = 3 if nf > 1500 else 5
    re, im = rng.standard_normal((2, rows, nf))
    im[0] *= 1e-12            # sizes far apart in one row
    re[1] = 0.0               # no real part: Im stays as it is
    gre, gim = ctx.kk(re, im, 0.0125)
    ere, eim = kk_longdouble(re, im)
    tol = 2 * max(nf, 8) * np.finfo(float).eps
    for got, want, row_scale in ((gre, ere, np.abs(re).max(1) + np.abs(im).max(1)),
                                 (gim, eim, np.abs(re).max(1) + np.abs(im).max(1))):
        err = np.abs(got.astype(np.longdouble) - want).max(1)
        assert (err <= tol * row_scale).all(), err / row_scale
    if nf <= 4096:
        assert np.array_equal(gim[1], im[1])


def test_kk_nonfinite_and_huge_rows(ctx):
    rng = np.random.default_rng(5)
    nf = 300
    re, im = rng.standard_normal((2, 5, nf))
    re[0, 7] = np.nan
    im[1, 9] = np.inf
    re[2, 3] = 1e300
    clean_re, clean_im = ctx.kk(re[3:], im[3:], 0.01)
    gre, gim = ctx.kk(re, im, 0.01)
    assert np.array_equal(gre[3:], clean_re) and np.array_equal(gim[3:], clean_im)
    # a NaN of Re reaches Im everywhere but at its own frequency, and Re only there
    assert np.isnan(np.delete(gim[0], 7)).all() and np.isfinite(gim[0, 7])
    assert np.isnan(gre[0, 7]) and np.isfinite(np.delete(gre[0], 7)).all()
    assert np.isinf(gre[1]).sum() == nf - 1 and np.isfinite(gim[1]).sum() == nf - 1
    assert np.isfinite(gre[2]).all() and np.isfinite(gim[2]).all()
