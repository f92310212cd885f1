"""A fixed eigensolver schedule holds for the adjoint too: its reduction is then the
one-stage one (other launches in the resolvent), with the same gradient."""
import numpy as np
import pytest

from test_oracle_grad import grad_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("encut,two_stage", [(110, True), (45, False)])
def test_adjoint_honours_schedule(ctx, tmp_path, encut, two_stage):
    import picomax_b200 as pm
    args, *_ = grad_case(tmp_path, soc=False, neps=4, nfreq=60, dfreq=0.2)
    args[args.index("-encut") + 1] = str(encut)
    p = pm.Problem(args)
    assert (p.info.npw >= 96) == two_stage
    chi = ctx.chi(p, pm.SWITCH_EPSLL, pm.PREC_FP64)
    rng = np.random.default_rng(3)
    gbar = rng.standard_normal((p.info.nq, p.info.nfreq)) + 1j * rng.standard_normal((p.info.nq, p.info.nfreq))
    grads, launches = [], []
    try:
        for schedule in (-1, 0, 1, 2):
            ctx.set_schedule(schedule)
            before = ctx.kernel_launches()
            grads.append(ctx.epsm_vjp(p, gbar, chi))
            launches.append(ctx.kernel_launches() - before)
    finally:
        ctx.set_schedule(-1)
    assert launches[0] == launches[1] and launches[2] == launches[3]
    assert (launches[1] != launches[2]) == two_stage
    # the same gradient from another reduction: n eps of the solver, and the oracle's 1e-8
    for g in grads[1:]:
        assert np.abs(g - grads[0]).max() <= 1e-8 * np.abs(grads[0]).max()
    p.close()
