"""The eigenvector adjoint on the two-stage reduction (n >= 96: Q^H by panels and
bulge-chasing reflectors, shifted tridiagonal solves) against the tangent-mode
oracle, padded and unpadded sizes, with and without spin-orbit coupling."""
import numpy as np
import pytest

import pmx_oracle as O
import pmx_oracle_grad as OG
from test_oracle_grad import grad_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soc,encut", [(True, 70), (False, 110), (True, 95)])
def test_epsm_vjp_two_stage_vs_oracle(ctx, tmp_path, soc, encut):
    import picomax_b200 as pm
    args, *_ = grad_case(tmp_path, soc=soc, neps=4, nfreq=60, dfreq=0.2)
    args[args.index("-encut") + 1] = str(encut)
    cr, mat, _, o = O.from_args(args)
    prob = pm.Problem(args)
    assert prob.info.npw * (2 if soc else 1) >= 96
    G, hkl = prob.gvectors()
    K, KW = prob.kpoints()
    Q = prob.qpoints()
    _, _, em, dem = OG.chi_ll_epsm(cr, mat, G, hkl, K, KW, Q, **o)
    rng = np.random.default_rng(11)
    gbar = rng.standard_normal(em.shape) + 1j * rng.standard_normal(em.shape)
    ref = np.einsum("pqf,qf->p", dem, gbar.conj()).real
    got = ctx.epsm_vjp(prob, gbar)
    assert np.max(np.abs(got - ref)) < 1e-8 * np.max(np.abs(ref))
    prob.close()
