"""Eigenvectors of tridiagonal matrices with many eigenvalues equal to rounding: chains
and graded matrices whose entries go down to 1e-150, in both solvers."""
import numpy as np
import pytest

from test_gpu_sturm_range import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["chain", "zeros", "diagonal", "graded"])
@pytest.mark.parametrize("n,nev", [(40, 40), (64, 20), (113, 113), (150, 30), (274, 274), (430, 60)])
def test_vectors_of_graded_matrices(ctx, kind, n, nev):
    rng = np.random.default_rng(7 * n + nev)
    mats = []
    for small in (1e-8, 1e-12, 1e-20, 1e-60, 1e-150):
        d, e = chain(rng, n, kind, small)
        mats.append((np.diag(d) + np.diag(e, 1) + np.diag(e, -1)).astype(complex))
    for schedule in (0, 1):
        ctx.set_schedule(schedule)
        try:
            w, z = ctx.heev(np.stack(mats), nev)
        finally:
            ctx.set_schedule(-1)
        for i, a in enumerate(mats):
            # a cluster of a hundred eigenvalues, many equal to rounding, keeps half the
            # digits at least: residual and orthogonality to sqrt(eps) (|A| <= 2)
            res = np.linalg.norm(a @ z[i] - z[i] * w[i], axis=0)
            orth = np.abs(z[i].conj().T @ z[i] - np.eye(nev))
            assert max(res.max(), orth.max()) <= np.sqrt(np.finfo(float).eps), (schedule, i, res.max(), orth.max())
