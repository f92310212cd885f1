"""The FP64 contraction's shares of the transitions (few tiles, many transitions:
contract64_split) and its kernel without the table of line shapes, against the oracle:
shares that end inside a chunk, that are empty because a narrow line leaves a tile fewer
chunks than shares, one and four channels."""
import numpy as np
import pytest

import pmx_oracle as O
import picomax_b200 as pm
from test_gpu_contract64 import GAAS, SI
from test_gpu_memory import give_back, leave

pytestmark = pytest.mark.gpu
SWITCH = {"epsLL": pm.SWITCH_EPSLL, "epsij": pm.SWITCH_EPSIJ}

# (crystal, switch, delta, epsilon, neps, nfreq, dfreq, nband, points). neps 1-3: one pair
# block and no table, 4-6: three blocks that share one; at least 256 transitions, two
# shares or more
CASES = [
    (SI, "epsLL", 1, 0.2, 1, 63, 0.4, 16, 17),     # 272: two shares over all frequencies
    (SI, "epsLL", 0, 0.002, 2, 130, 0.2, 16, 29),  # a line narrower than a step
    (SI, "epsLL", 1, 0.2, 4, 64, 0.4, 16, 33),     # 528, table
    (SI, "epsLL", 0, 0.004, 6, 130, 0.2, 16, 65),  # 1040, table, sparse tiles
    (GAAS, "epsij", 1, 0.01, 3, 127, 0.2, 13, 11),  # four channels, windows of epsij
    (GAAS, "epsij", 0, 0.02, 4, 65, 0.3, 14, 23),   # 1104, table
]


def case(i, tmp_path, **change):
    base, sw, delta, eps, neps, nf, df, nband, nk = CASES[i]
    rng = np.random.default_rng(300 + i)
    K = rng.uniform(-0.4, 0.4, (nk, 3))
    kf = str(tmp_path / "k.txt")
    pm.write_kfile(kf, K, rng.uniform(0.5, 1.5, nk))
    opt = {"neps": neps, "nband": nband, "nfreq": nf, "dfreq": df, "delta": delta, "epsilon": eps, **change}
    return K, opt, base + ["-encut", "45", "-switch", sw, "-kpoint", "0", "-kpointfile", kf, "-qvec",
                           "0.03,0.01,0.02", "-nvalence", "8", "-kk", "1"] + [str(x) for kv in opt.items() for x in
                                                                              ("-" + kv[0], kv[1])]


@pytest.mark.parametrize("i", range(len(CASES)))
def test_shares_vs_oracle(ctx, tmp_path, i):
    K, opt, args = case(i, tmp_path)
    p = pm.Problem(args)
    G, hkl = p.gvectors()
    cr, mat, _, _ = O.from_args(args)
    re, im = O.chi(cr, mat, G, hkl, K, p.kpoints()[1], p.qpoints(), mode=CASES[i][1], nvalence=8, kk=1, **opt)
    gre, gim = ctx.chi(p, SWITCH[CASES[i][1]], pm.PREC_FP64)
    scale = max(np.abs(re).max(), np.abs(im).max())
    assert scale > 0
    assert np.abs(gre - re.ravel()).max() < 1e-8 * scale and np.abs(gim - im.ravel()).max() < 1e-8 * scale
    p.close()


@pytest.mark.parametrize("mb", [75, 48])
@pytest.mark.parametrize("i", [2, 3, 5])
def test_without_the_table(tmp_path, i, mb):
    """The same spectrum on a fine grid where the allocation of the table fails, and that
    of the shares' partial sums."""
    _, _, small = case(i, tmp_path)
    _, _, args = case(i, tmp_path, neps=4, nfreq=8000, dfreq=0.004, delta=1, epsilon=0.2)
    sw = SWITCH[CASES[i][1]]
    if sw == pm.SWITCH_EPSIJ:  # a window of 50 epsilon: the whole grid
        args[args.index("-epsilon") + 1] = "0.7"
    p, ps = pm.Problem(args), pm.Problem(small)
    c = pm.Context(0)
    want = c.chi(p, sw, pm.PREC_FP64)
    c.close()
    c = pm.Context(0)
    held = []
    try:
        c.chi(ps, sw, pm.PREC_FP64)  # loads the kernels
        # acc, chi and chi2: 18 x 10 x 8000 doubles each, 35 MB, 23 MB for two shares of acc;
        # the table 1 MB for every 16 transitions: 34, 66, 70 MB
        held.append(leave(mb))
        got = c.chi(p, sw, pm.PREC_FP64)
    finally:
        c.close()
        give_back(held)
    for g, w in zip(got, want):
        # the line shape from another place in the code: its rounding, summed
        assert np.abs(g - w).max() <= 1e-13 * np.abs(w).max()
    p.close()
    ps.close()
