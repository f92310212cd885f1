"""Calls on a device with little memory left: the workspaces sized for speed (a group of
q's eigenproblems, the table of line shapes kept from an earlier call) are given back and
the call runs with small ones, with the same result."""
import numpy as np
import pytest

import picomax_b200 as pm
from picomax_b200.kgrid import gamma_grid

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SI = ["-crystal", "zb", "-a", "5.43", "-vg", "3,4,8,11,-0.21,0,0.04,0.08,-0.21,0,0.04,0.08", "-encut", "110",
      "-kpoint", "0", "-nband", "16", "-nvalence", "8", "-dfreq", "0.1", "-epsilon", "0.2", "-kk", "1"]
MB = 1 << 20


def problem(tmp_path, name, K, **kw):
    kf = str(tmp_path / name)
    pm.write_kfile(kf, K, np.ones(len(K)))
    return pm.Problem(SI + ["-switch", "epsLL", "-kpointfile", kf] + [str(x) for kv in kw.items() for x in
                                                                     ("-" + kv[0], kv[1])])


def leave(mb):
    """Takes the device's memory but for mb MB."""
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    assert free > mb * MB
    return torch.empty(free - mb * MB, dtype=torch.uint8, device="cuda")


def give_back(held):
    held.clear()
    torch.cuda.empty_cache()


def close_to(a, b):
    return all(np.abs(x - y).max() <= 1e-9 * np.abs(y).max() for x, y in zip(a, b))


def test_group_of_q_that_does_not_fit(tmp_path):
    """8 k and 150 q: one solve of 1192 matrices of 128 x 128 (0.6 GB with reflectors,
    scratch and vectors), or 150 of 8."""
    rng = np.random.default_rng(1)
    q = ",".join(f"{x:.4f}" for x in rng.uniform(0.01, 0.3, 450))
    p = problem(tmp_path, "k.txt", rng.uniform(-0.4, 0.4, (8, 3)), neps=3, nfreq=64, delta=0, qvec=q)
    c = pm.Context(0)
    want = c.chi(p, pm.SWITCH_EPSLL, pm.PREC_FP64)
    c.close()
    held = [leave(300)]
    c = pm.Context(0)
    try:
        got = c.chi(p, pm.SWITCH_EPSLL, pm.PREC_FP64)
        assert close_to(got, want)
        assert torch.cuda.mem_get_info()[0] < 300 * MB
    finally:
        c.close()
        give_back(held)


def test_table_kept_from_an_earlier_call(tmp_path):
    """A first call whose table of line shapes takes 0.3 GB, then a smaller one whose
    spectra do not fit beside it."""
    K, _ = gamma_grid("zb", 8, 8, 8)
    first = problem(tmp_path, "k1.txt", K, neps=4, nfreq=4000, delta=1, qvec="0.05,0.01,0.02")
    second = problem(tmp_path, "k2.txt", K[:9] + 0.01, neps=20, nfreq=2000, delta=1, qvec="0.05,0.01,0.02")
    c = pm.Context(0)
    want = c.chi(second, pm.SWITCH_EPSLL, pm.PREC_FP64)
    c.close()
    c = pm.Context(0)
    held = []
    try:
        c.chi(first, pm.SWITCH_EPSLL, pm.PREC_FP64)
        held.append(leave(100))
        got = c.chi(second, pm.SWITCH_EPSLL, pm.PREC_FP64)
        assert close_to(got, want)
    finally:
        c.close()
        give_back(held)


def test_adjoint_and_bands(tmp_path):
    """The adjoint's blocks of k-points (1.5 GB in one, 0.3 GB) shrink as well."""
    K, _ = gamma_grid("zb", 12, 12, 12)
    p = problem(tmp_path, "k.txt", K + 0.003, neps=3, nfreq=64, delta=0, qvec="0.05,0.01,0.02")
    nf = 64
    rng = np.random.default_rng(2)
    results = []
    held = []
    try:
        for mb in (None, 450):
            c = pm.Context(0)
            if mb:
                held.append(leave(mb))
            band = c.band(p)
            re, im, eps = c.chi_epsm(p, pm.SWITCH_EPSLL, pm.PREC_FP64)
            g = results[0][-1] if results else rng.standard_normal((1, nf)) + 1j * rng.standard_normal((1, nf))
            grad = c.epsm_vjp(p, g, (re, im))
            results.append((band, eps.view(float), grad, g))
            c.close()
    finally:
        give_back(held)
    for a, b in zip(results[1][:3], results[0][:3]):
        assert np.abs(a - b).max() <= 1e-7 * np.abs(b).max()


def test_out_of_memory_is_an_error_and_no_more(tmp_path):
    """A call that fits in no way fails, and the context works afterwards."""
    K, _ = gamma_grid("zb", 2, 2, 2)
    big = problem(tmp_path, "k1.txt", K, neps=20, nfreq=4000, delta=0, qvec="0.05,0.01,0.02")
    small = problem(tmp_path, "k2.txt", K, neps=2, nfreq=16, delta=0, qvec="0.05,0.01,0.02")
    c = pm.Context(0)
    want = c.chi(small, pm.SWITCH_EPSLL, pm.PREC_FP64)
    held = [leave(60)]
    try:
        with pytest.raises(pm.PicomaxError):
            c.chi(big, pm.SWITCH_EPSLL, pm.PREC_FP64)
        got = c.chi(small, pm.SWITCH_EPSLL, pm.PREC_FP64)
        assert close_to(got, want)
    finally:
        c.close()
        give_back(held)
