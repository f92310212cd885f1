"""An eigensolver error names the set of the common solve that its matrix belongs to:
reference point, q-point of a band, k-point, k-point of k + q."""
import numpy as np
import pytest

import picomax_b200 as pm

pytestmark = pytest.mark.gpu

SI = ["-crystal", "zb", "-a", "5.43", "-vg", "3,4,8,11,-0.21,0,0.04,0.08,-0.21,0,0.04,0.08", "-encut", "45"]


def chi_args(tmp_path, K, q):
    kf = str(tmp_path / "k.txt")
    pm.write_kfile(kf, np.asarray(K, float), np.ones(len(K)))
    return SI + ["-switch", "epsLL", "-kpoint", "0", "-kpointfile", kf, "-qvec", q, "-neps", "2", "-nband", "12",
                 "-nvalence", "8", "-nfreq", "16", "-dfreq", "0.5", "-delta", "0", "-epsilon", "0.3", "-kk", "1"]


def message(call):
    with pytest.raises(pm.PicomaxError) as e:
        call()
    assert e.value.status == pm.PMX_ERR_NOCONV
    return str(e.value)


def test_names(tmp_path):
    K = [[0.1, 0.2, 0.05], [0.15, -0.1, 0.3]]
    p = pm.Problem(chi_args(tmp_path, K, "0.02,0.01,0.03,nan,0,0"))
    c = pm.Context(0)
    text = message(lambda: c.chi(p, pm.SWITCH_EPSLL))
    assert "at k + q (q 1), k-point 0" in text
    text = message(lambda: c.epsm_vjp(p, np.ones((2, 16), complex), (np.zeros(p.info.chi_values),) * 2))
    assert "at k + q (q 1), k-point 0 + 0" in text
    c.set_fault(2)  # every bisection is cut short: the first matrix of the solve reports
    assert "at reference point 0" in message(lambda: c.chi(p, pm.SWITCH_EPSLL))
    c.set_fault(0)
    p.close()
    p = pm.Problem(chi_args(tmp_path, [K[0], [1e200, 0, 0]], "0.02,0.01,0.03"))
    assert "at k-point 1" in message(lambda: c.chi(p, pm.SWITCH_EPSLL))
    p.close()
    p = pm.Problem(SI + ["-switch", "band", "-nband", "8", "-nvalence", "8", "-qvec", "0,0,0,nan,0,0"])
    assert "at q-point 1" in message(lambda: c.band(p))
    p.close()
    c.close()
