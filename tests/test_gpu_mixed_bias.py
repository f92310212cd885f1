"""FP32 sums of the mixed contraction (mixed.cu): their bias where thousands of
transitions of one frequency stand together, and their division of a transition list
of any length into pairs of interleaved sums."""
import numpy as np
import pytest

import picomax_b200 as pm
from picomax_b200.workloads import workload

pytestmark = pytest.mark.gpu

SI = ["-crystal", "zb", "-a", "5.43", "-vg", "3,4,8,11,-0.21,0,0.04,0.08,-0.21,0,0.04,0.08"]
GAAS = ["-crystal", "zb", "-a", "5.65", "-vg", "3,4,8,11,-0.23,-0.2,0.01,0.06,-0.2,0.07,0.05,0.01", "-ua_so",
        "3:0.002,4:0.003,8:0.001", "-use_uniform_us_so", "-uniform_us_so_val", "0.004"]


def test_bias_of_dense_spectrum(ctx, tmp_path):
    """Wurtzite, 9216 k: about 300 transitions under one line. In one FP32 sum they cost
    60 additions of half a unit in the last place (2^-24 of a sum that is half full on
    average, and as much again for the products): 4e-6. Spread over the sums of an item
    no sum has more than a few, which leaves the rounding of the BF16 operands (2^-17,
    random): 1e-6 with room."""
    args, *_ = workload("wz_epsLL", str(tmp_path))
    p = pm.Problem(args)
    ref = ctx.chi(p, pm.SWITCH_EPSLL, pm.PREC_FP64)
    ctx.set_overlap_mode(0)  # FP64 overlaps: the contraction's own error
    try:
        got = ctx.chi(p, pm.SWITCH_EPSLL, pm.PREC_MIXED)
    finally:
        ctx.set_overlap_mode(1)
    for g, r in zip(got, ref):
        assert np.linalg.norm(g - r) <= 1e-6 * np.linalg.norm(r)
    p.close()


@pytest.mark.parametrize("nk", [1, 5, 33, 90, 400])
@pytest.mark.parametrize("base,sw,delta", [(SI, "epsLL", 0), (SI, "epsLL", 1), (GAAS, "epsij", 0)])
def test_every_transition_once(ctx, tmp_path, base, sw, delta, nk):
    """Lists from below one chunk to several blocks of sums, windows of zero line shape,
    all frequencies and windows of epsij: a transition lost, doubled or of the wrong sign
    among at most 40 000 shows in the spectrum (2e-5 of it)."""
    rng = np.random.default_rng(nk)
    kf = str(tmp_path / "k.txt")
    pm.write_kfile(kf, rng.uniform(-0.4, 0.4, (nk, 3)), rng.uniform(0.5, 1.5, nk))
    p = pm.Problem(base + ["-encut", "45", "-switch", sw, "-kpoint", "0", "-kpointfile", kf, "-qvec", "0.03,0.01,0.02",
                           "-neps", "3", "-nband", "13", "-nvalence", "8", "-nfreq", "300", "-dfreq", "0.05",
                           "-delta", str(delta), "-epsilon", "0.1", "-kk", "1"])
    switch = pm.SWITCH_EPSLL if sw == "epsLL" else pm.SWITCH_EPSIJ
    ref = np.concatenate([x.ravel() for x in ctx.chi(p, switch, pm.PREC_FP64)])
    got = np.concatenate([x.ravel() for x in ctx.chi(p, switch, pm.PREC_MIXED)])
    assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)
    p.close()
