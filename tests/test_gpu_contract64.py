"""The FP64 tensor-core contraction (contract64.cu) and the windows of zero line
shape against the numpy oracle, at the edges of its tiles: 3 local-field vectors
per block, 64 frequencies, 16 transitions, shares of the transitions."""
import numpy as np
import pytest

import pmx_oracle as O

pytestmark = pytest.mark.gpu

SI = ["-crystal", "zb", "-a", "5.43", "-vg", "3,4,8,11,-0.21,0,0.04,0.08,-0.21,0,0.04,0.08"]
GAAS = ["-crystal", "zb", "-a", "5.65", "-vg", "3,4,8,11,-0.23,-0.2,0.01,0.06,-0.2,0.07,0.05,0.01", "-ua_so",
        "3:0.002,4:0.003,8:0.001", "-use_uniform_us_so", "-uniform_us_so_val", "0.004"]

# (crystal, switch, delta, epsilon, neps, nfreq, dfreq, nband, points): widths of
# the line shape from under one step to beyond the grid (dense), 1 and 4 channels
CASES = [
    (SI, "epsLL", 0, 0.02, 1, 63, 0.4, 12, 1),
    (SI, "epsLL", 0, 0.1, 3, 65, 0.4, 16, 3),
    (SI, "epsLL", 0, 0.004, 4, 300, 0.1, 12, 5),
    (SI, "epsLL", 1, 0.2, 7, 129, 0.2, 12, 2),
    (SI, "epsLL", 2, 0.5, 9, 64, 0.4, 12, 2),
    (SI, "epsLL", 3, 0.9, 2, 191, 0.15, 20, 3),
    (SI, "epsij", 0, 0.1, 5, 128, 0.2, 12, 2),
    (GAAS, "epsij", 1, 0.02, 3, 127, 0.2, 14, 2),
    (GAAS, "epsij", 2, 0.6, 4, 64, 0.3, 12, 1),
    (GAAS, "epsLL", 0, 0.05, 6, 97, 0.3, 13, 2),
    (GAAS, "epsxyz", 0, 0.05, 3, 66, 0.3, 12, 2),
]


@pytest.mark.parametrize("i", range(len(CASES)))
def test_contraction_vs_oracle(ctx, tmp_path, i):
    import picomax_b200 as pm
    base, sw, delta, eps, neps, nf, df, nband, nk = CASES[i]
    rng = np.random.default_rng(100 + i)
    K = rng.uniform(-0.4, 0.4, (nk, 3))
    kf = str(tmp_path / "k.txt")
    pm.write_kfile(kf, K, np.ones(nk))
    args = base + ["-encut", "45", "-switch", sw, "-kpoint", "0", "-kpointfile", kf, "-qvec", "0.03,0.01,0.02",
                   "-neps", str(neps), "-nband", str(nband), "-nvalence", "8", "-nfreq", str(nf), "-dfreq", str(df),
                   "-delta", str(delta), "-epsilon", str(eps), "-kk", "1"]
    p = pm.Problem(args)
    G, hkl = p.gvectors()
    cr, mat, _, o = O.from_args(args)
    kw = dict(neps=neps, nband=nband, nvalence=8, nfreq=nf, dfreq=df, epsilon=eps, delta=delta, kk=1)
    W = p.kpoints()[1]
    if sw == "epsxyz":
        re, im = O.chi_xyz(cr, mat, G, hkl, K, W, p.qpoints(), **kw)
    else:
        re, im = O.chi(cr, mat, G, hkl, K, W, p.qpoints(), mode=sw, **kw)
    switch = {"epsLL": pm.SWITCH_EPSLL, "epsij": pm.SWITCH_EPSIJ, "epsxyz": pm.SWITCH_EPSXYZ}[sw]
    for precision, tol in ((pm.PREC_FP64, 1e-8), (pm.PREC_MIXED, 1e-4)):
        gre, gim = ctx.chi(p, switch, precision)
        scale = max(np.abs(re).max(), np.abs(im).max())
        assert scale > 0
        assert np.abs(gre - re.ravel()).max() < tol * scale
        assert np.abs(gim - im.ravel()).max() < tol * scale
