"""eps_M at and beside its poles, where the block of the local-field vectors without
vector 0 is singular: [eps^-1]_00 is zero there (eps_M infinite, the loss function
zero) although eps itself is regular."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spectra(neps, j, deltas, seed):
    """chi of one q whose eps has row and column j zero but for eps_jj = deltas[f] and
    the coupling to vector 0: [eps^-1]_00 = 0 where delta = 0. Returns re, im, eps."""
    rng = np.random.default_rng(seed)
    nf = len(deltas)
    eps = np.zeros((nf, neps, neps), complex)
    for f, d in enumerate(deltas):
        a = rng.standard_normal((neps, neps)) + 1j * rng.standard_normal((neps, neps))
        a = 0.3 * (a + a.conj().T) / np.sqrt(neps) + 2 * np.eye(neps)
        a[0, 0] += 0.5j  # a complex diagonal, as absorption makes it
        c = a[j, 0] if neps > 2 else 0.7 + 0.2j
        a[j, 1:] = a[1:, j] = 0.0
        a[j, j] = d
        a[j, 0], a[0, j] = c, np.conj(c)
        eps[f] = a
    tri = [(m, n) for m in range(neps) for n in range(m + 1)]
    chi = np.stack([eps[:, m, n] - (1.0 if m == n else 0.0) for m, n in tri])[None]
    for m, n in tri:  # what the device adds again is exact
        if m == n:
            eps[:, m, m] = chi[0, tri.index((m, m))] + 1.0
    return np.ascontiguousarray(chi.real), np.ascontiguousarray(chi.imag), eps


@pytest.mark.parametrize("neps", [2, 3, 16, 17, 33, 64])
def test_epsm_at_poles(ctx, neps):
    deltas = [0.0, 2.0 ** -40, 0.0, -(2.0 ** -50), 1.0]
    for j in sorted({1, neps // 2, neps - 1} - {0}):
        re, im, eps = spectra(neps, j, deltas, 10 * neps + j)
        got = ctx.eps_macroscopic(neps, re, im)[0]
        for f, d in enumerate(deltas):
            if d == 0.0:
                assert np.isposinf(got[f].real) and got[f].imag == 0.0, (j, got[f])
                continue
            # 1 / eps_M: elimination is backward stable, n eps |eps^-1|
            want = np.linalg.inv(eps[f])
            tol = neps * np.finfo(float).eps * np.linalg.norm(want, 2) * np.linalg.cond(eps[f])
            assert abs(1.0 / got[f] - want[0, 0]) <= tol, (j, d)
        loss, _ = ctx.eels(got[None], 0.1)
        assert np.isfinite(loss).all() and loss[0, 0] == 0.0 and loss[0, 2] == 0.0


def test_epsm_singular_and_nan(ctx):
    """eps itself singular (its last pivot vanishes) stays zero, NaN stays NaN."""
    re = np.array([[[-1.0, np.nan], [0.0, 0.1], [0.0, 0.2]]])  # eps_00, eps_10, eps_11 - 1
    got = ctx.eps_macroscopic(2, re, np.zeros_like(re))[0]
    assert got[0] == 0.0 and np.isnan(got[1])
