"""Scaling of a row's two halves in the FFT Kramers-Kronig transform (kk_fft.cu): an
entry 0 of any size (its weight is zero), and halves of very different size, whose
sums are looked at where the other half is zero."""
import numpy as np
import pytest

from test_gpu_kk_fft import kk_longdouble

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


# what the sum over an array of norm |x| may be off by: the transform's
# log2(L) <= 13 stages of eps |x| each, and the rounding of the final sum
def bound(x, out):
    norm = np.sqrt((np.abs(x).astype(np.longdouble) ** 2).sum())  # squares of 1e-200 leave the FP64 range
    return 32 * EPS * norm + 2 * EPS * np.abs(out)


@pytest.mark.parametrize("big", [1e12, -1e200, 1e305])
@pytest.mark.parametrize("nf", [2, 65, 1000, 4096])
def test_kk_entry_zero_has_no_weight(ctx, nf, big):
    rng = np.random.default_rng(nf)
    y = rng.standard_normal(nf)
    x = np.zeros(nf)
    x[0] = big
    re, im = np.stack([x, y]), np.stack([y, x])
    gre, gim = ctx.kk(re, im, 0.0125)
    ere, eim = kk_longdouble(np.stack([0 * x, y]), np.stack([y, 0 * x]))
    # nothing is added to y: the other half's only entry has no weight
    assert np.array_equal(gim[0], y) and np.array_equal(gre[1], y)
    # the sum over y, at every frequency but 0 (where the large entry itself stands)
    y0 = y.copy()
    y0[0] = 0.0
    for got, want in ((gre[0], ere[0]), (gim[1], eim[1])):
        err = np.abs(got[1:].astype(np.longdouble) - want[1:])
        assert (err <= bound(y0, want[1:])).all(), err.max()
        assert got[0] == big or abs(big) < 1e13


@pytest.mark.parametrize("nf", [65, 1000, 4096])
def test_kk_entry_zero_beside_small_rest(ctx, nf):
    rng = np.random.default_rng(nf + 1)
    re, im = rng.standard_normal((2, 1, nf)) * 1e-6
    with_big = re.copy()
    with_big[0, 0] = 1e10
    gre, gim = ctx.kk(with_big, im, 0.0125)
    cre, cim = ctx.kk(re, im, 0.0125)
    assert np.array_equal(gre[0, 1:], cre[0, 1:]) and np.array_equal(gim, cim)


@pytest.mark.parametrize("ratio", [1e-12, 1e-200])
@pytest.mark.parametrize("nf", [64, 1000, 4096])
def test_kk_halves_of_different_size(ctx, nf, ratio):
    rng = np.random.default_rng(nf + 2)
    re, im = np.zeros((2, 1, nf))
    re[0, :nf // 2] = rng.standard_normal(nf // 2)      # large, zero in the upper half
    im[0] = ratio * rng.standard_normal(nf)
    for a, b, swap in ((re, im, False), (im, re, True)):
        ga, gb = ctx.kk(a, b, 0.0125)
        if swap:
            ga, gb = gb, ga
        ere, eim = kk_longdouble(re, im)
        # Re out = Re + sum over the small Im, seen where Re is zero
        err = np.abs(ga[0, nf // 2:].astype(np.longdouble) - ere[0, nf // 2:])
        assert (err <= bound(im, ere[0, nf // 2:])).all(), err.max()
        err = np.abs(gb[0].astype(np.longdouble) - eim[0])
        assert (err <= bound(re, eim[0])).all(), err.max()
