"""eps_M on the device against the numpy inverse for every number of warps and at
the edges of its lane passes (1 .. 64 local-field vectors)."""
import numpy as np
import pytest

import pmx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neps", [1, 2, 3, 15, 16, 17, 31, 32, 33, 34, 59, 64])
def test_epsm_sizes(ctx, neps):
    rng = np.random.default_rng(neps)
    npair, nf, nq = neps * (neps + 1) // 2, 5, 2
    re, im = 0.4 * rng.standard_normal((2, nq, npair, nf)) / np.sqrt(neps)
    got = ctx.eps_macroscopic(neps, re, im)
    for q in range(nq):
        want = O.eps_macroscopic(re[q], im[q], neps)
        # a matrix of order n, condition below 1e4: n eps cond
        assert np.abs(got[q] - want).max() < 1e-10 * np.abs(want).max()
