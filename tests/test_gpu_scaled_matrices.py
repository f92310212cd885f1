"""Hermitian matrices in any unit: eigenvalues relative to the norm and eigenvectors do
not depend on a common factor of the matrix, in both solvers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALES = [1e-140, 1e-6, 1.0, 1e3, 1e6, 1e10, 1e100, 1e150]


@pytest.mark.parametrize("schedule", [0, 1])
@pytest.mark.parametrize("n,nev", [(64, 9), (96, 20), (113, 113), (150, 30), (274, 17), (430, 12), (850, 6)])
def test_common_factor(ctx, n, nev, schedule):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a = (a + a.conj().T) / 2
    a /= np.linalg.norm(a, 2)
    want = np.linalg.eigvalsh(a)[:nev]
    ctx.set_schedule(schedule)
    try:
        w, z = ctx.heev(np.stack([s * a for s in SCALES]), nev)
    finally:
        ctx.set_schedule(-1)
    eps = np.finfo(float).eps
    for i, s in enumerate(SCALES):
        # backward stable reductions: a small multiple of n eps |A|
        assert np.abs(w[i] / s - want).max() <= n * eps, s
        res = np.linalg.norm(a @ z[i] - z[i] * (w[i] / s), axis=0)
        assert res.max() <= 10 * n * eps, s
        assert np.abs(z[i].conj().T @ z[i] - np.eye(nev)).max() <= 1e-11, s
