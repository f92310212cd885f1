"""Length of the FP32 sums of the mixed contraction (mixed.cu) where the
frequencies of zero line shape are left out and a frequency's transitions stand
together: Te + SOC, 18 x 6 bands, thousands of transitions per line."""
import numpy as np
import pytest

import picomax_b200 as pm
from picomax_b200.workloads import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epsilon", ["0.05", "0.2"])
def test_mixed_sums_stay_short(ctx, tmp_path, epsilon):
    args, *_ = workload("te_epsLL", str(tmp_path))
    args = list(args)
    if "-epsilon" in args:
        args[args.index("-epsilon") + 1] = epsilon
    else:
        args += ["-epsilon", epsilon]
    p = pm.Problem(args)
    ref = np.concatenate([x.ravel() for x in ctx.chi(p, pm.SWITCH_EPSLL, pm.PREC_FP64)])
    got = np.concatenate([x.ravel() for x in ctx.chi(p, pm.SWITCH_EPSLL, pm.PREC_MIXED)])
    # 16 chunks of 6 products: 96 additions to a sum that is half full on average,
    # each at most one unit in the last place (2^-23) short
    assert np.linalg.norm(got - ref) <= 48 * 2.0**-23 * np.linalg.norm(ref)
