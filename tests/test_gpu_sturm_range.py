"""Sturm counts of tridiagonal matrices whose entries span the FP64 range: chains with a
zero diagonal, a probe exactly at it, and off-diagonals down to 1e-150, with and without
exact zeros among them, in both solvers (a tridiagonal input passes the reductions as it
is)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(rng, n, kind, small):
    e = rng.uniform(0.2, 1.0, n - 1) * np.where(rng.random(n - 1) < 0.4, small, 1.0)
    d = np.zeros(n)
    if kind == "zeros":
        e[rng.random(n - 1) < 0.2] = 0.0
    if kind == "diagonal":
        d = np.where(rng.random(n) < 0.5, small, 0.0)
        e[rng.random(n - 1) < 0.5] = 0.0
    if kind == "graded":
        e *= np.logspace(0, np.log10(small), n - 1)
    return d, e


@pytest.mark.parametrize("kind", ["chain", "zeros", "diagonal", "graded"])
@pytest.mark.parametrize("n,nev", [(40, 40), (64, 21), (113, 113), (150, 150), (150, 85), (274, 274), (300, 60)])
def test_sturm_counts_in_range(ctx, kind, n, nev):
    rng = np.random.default_rng(n + nev)
    mats, want = [], []
    for small in (1e-20, 1e-40, 1e-60, 1e-95, 1e-150):
        d, e = chain(rng, n, kind, small)
        a = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
        mats.append(a.astype(complex))
        want.append(np.linalg.eigvalsh(a)[:nev])
    for schedule in (0, 1):
        ctx.set_schedule(schedule)
        try:
            w, _ = ctx.heev(np.stack(mats), nev, vectors=False)
        finally:
            ctx.set_schedule(-1)
        for i in range(len(mats)):
            # eigvalsh's own n eps |A| (|A| <= 2)
            assert np.abs(np.sort(w[i]) - want[i]).max() <= 2 * n * np.finfo(float).eps, (schedule, i)
