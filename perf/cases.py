"""Performance cases of picomax_b200: what a user of the library has it do, with sizes, inputs and work.

Every case runs through the package's public entry points (Context / Problem
methods and the torch autograd wrappers) on inputs drawn from a seed. The
crystals are those of picomax_b200.workloads; a seed moves their form factors
by a few per cent (as a fit or a convergence study does) and shifts the k grid
off the symmetry points, so that no band window cuts a degenerate set and every
output is determined by its input. One device context serves the whole process,
as in a user's program.

Kinds of cases:
  band   the band structure along a path (Context.band)
  chi    the susceptibility of one or more q with the spectra left on the GPU
         (Context.chi_device), in FP64 or mixed precision; mixed spectra, whose
         stated accuracy is 1e-4, are kept in single precision
  line   eps_M and the loss function along a line of q in FP64 (the loss is
         sensitive near the zeros of eps_M): plasmon dispersion
         (Context.chi_epsm without chi, then Context.eels)
  batch  eps_M of several crystals of uneven size, metals among them, in merged
         launches (Context.chi_batch), FP64
  fit    one training step on bands and eps_M: forward and backward through the
         hand-written adjoint (picomax_b200.autograd)
  post   post-processing of a spectrum loaded from a file: Kramers-Kronig,
         eps_M, loss function, all on host arrays (Context.kk,
         Context.eps_macroscopic, Context.eels)
"""
import math
import os
import tempfile

import numpy as np
import torch

import picomax_b200 as pm
from picomax_b200 import autograd as pmad
from picomax_b200 import workloads as wl

KCON = 3.809982111485962       # hbar^2 / 2m, eV A^2
RY = 13.605699169854621        # eV
ESU, EV, EM, HBAR = 4.803204712570263e-10, 1.602176634e-12, 9.1093837015e-28, 1.054571817e-27
_DEV = "cuda"
MIXED_TYPES = (torch.float32, torch.complex64)

# preset, lattice constant, c/a, u of the workloads' crystals
CRYSTALS = {
    "si": ("zb", 5.43, None, None),
    "gaas": ("zb", 5.65, None, None),
    "wz": ("wz", 3.19, 1.626, 0.375),
    "te": ("te", 4.45, 1.33, 0.264),
}
PATHS = {"zb": "G,X,W,L,G", "wz": "G,A,H,K,G", "te": "G,A,H,K,G"}

# local-field vectors (h k l) in the order of the library's G list, which decides how eps_M fills the matrix from its
# stored half; vectors of equal length have no order of their own
_ORDER = {
    ("si", 110): (
        "0,0,0 0,0,1 0,1,0 -1,-1,-1 1,1,1 0,-1,0 0,0,-1 1,0,0 -1,0,0 0,1,1 1,1,0 -1,0,-1 1,0,1 0,-1,-1 "
        "-1,-1,0 -1,0,1 1,0,-1 -1,1,0 -1,-1,-2 0,-1,1 1,-1,0 -2,-1,-1 2,1,1 1,1,2 -1,-2,-1 1,2,1 0,1,-1"),
    ("gaas", 120): (
        "0,0,0 0,-1,0 1,0,0 0,0,-1 0,0,1 1,1,1 0,1,0 -1,-1,-1 -1,0,0 -1,-1,0 0,-1,-1 1,0,1 1,1,0 0,1,1 "
        "-1,0,-1 -1,-2,-1 1,2,1 0,-1,1 1,0,-1 -2,-1,-1 1,1,2 1,-1,0 0,1,-1 -1,-1,-2 2,1,1 -1,0,1 -1,1,0"),
    ("wz", 260): (
        "0,0,0 0,0,1 0,0,-1 1,0,0 -1,0,0 1,-1,0 0,-1,0 -1,1,0 0,1,0 0,0,-2 0,0,2 0,1,1 -1,0,-1 -1,0,1 0,-1,1 "
        "1,0,-1 0,1,-1 1,0,1 0,-1,-1 1,-1,-1 -1,1,1 1,-1,1 -1,1,-1 0,-1,2 1,0,-2 -1,1,2 -1,0,-2 1,0,2 0,-1,-2 "
        "0,1,-2 -1,0,2 1,-1,2 1,-1,-2 0,1,2 -1,1,-2 0,0,-3 0,0,3 -1,-1,0 1,1,0 1,-2,0 2,-1,0 -2,1,0 -1,2,0 "
        "1,1,-1 1,1,1 -1,-1,1 -1,-1,-1 -2,1,1 -2,1,-1 -1,2,-1 -1,2,1 1,-2,-1 2,-1,1 1,-2,1 2,-1,-1 0,-1,3 "
        "0,-1,-3 1,0,3 -1,0,3"),
    ("te", 120): (
        "0,0,0 0,0,-1 0,0,1 1,-1,0 -1,1,0 0,1,0 0,-1,0 -1,0,0 1,0,0 0,1,1 0,1,-1 -1,0,1 1,0,1 1,0,-1 -1,0,-1"),
}


def listed():
    return [
        # band structure of a small cell: the first thing a user runs, 122 small matrices (n 113): latency
        dict(name="band_si_path", kind="band", crystal="si", encut=110, points=120, nband=16, nvalence=8),
        # the same of a spin-orbit crystal with large matrices (n 570) that nearly fill one wave of SMs
        dict(name="band_te_path", kind="band", crystal="te", encut=120, points=120, nband=24, nvalence=18),
        # the small silicon configuration, dense Gaussian spectra in FP64 (the CLI's default precision)
        dict(name="chi_si_ll_fp64", kind="chi", crystal="si", switch="epsLL", precision="fp64", encut=110, n1=8, n2=8,
             n3=8, nq=1, neps=15, nband=16, nvalence=8, nfreq=1000, dfreq=0.02, delta=0, epsilon=0.1, kk=1),
        # the GaAs + spin-orbit tensor configuration (Lorentzian, windowed) in FP64 on a convergence-test grid
        dict(name="chi_gaas_ij_fp64", kind="chi", crystal="gaas", switch="epsij", precision="fp64", encut=120, n1=6,
             n2=6, n3=6, nq=1, neps=27, nband=16, nvalence=8, nfreq=2000, dfreq=0.0125, delta=1, epsilon=0.05, kk=1),
        # the same at its full 16^3 grid in mixed precision: the headline spectrum
        dict(name="chi_gaas_ij_mixed", kind="chi", crystal="gaas", switch="epsij", precision="mixed", encut=120,
             n1=16, n2=16, n3=16, nq=1, neps=27, nband=16, nvalence=8, nfreq=2000, dfreq=0.0125, delta=1,
             epsilon=0.05, kk=1),
        # the wurtzite configuration (N_G 401, 59 local-field vectors) in mixed precision, half its grid per axis
        dict(name="chi_wz_ll_mixed", kind="chi", crystal="wz", switch="epsLL", precision="mixed", encut=260, n1=12,
             n2=12, n3=8, nq=1, neps=59, nband=48, nvalence=16, nfreq=2000, dfreq=0.015, delta=0, epsilon=0.1, kk=1),
        # its FP64 reference run on a coarse grid
        dict(name="chi_wz_ll_fp64", kind="chi", crystal="wz", switch="epsLL", precision="fp64", encut=260, n1=6, n2=6,
             n3=4, nq=1, neps=59, nband=48, nvalence=16, nfreq=2000, dfreq=0.015, delta=0, epsilon=0.1, kk=1),
        # trigonal tellurium with spin-orbit coupling: few k-points, large matrices
        dict(name="chi_te_ll_fp64", kind="chi", crystal="te", switch="epsLL", precision="fp64", encut=120, n1=6, n2=6,
             n3=5, nq=1, neps=15, nband=24, nvalence=18, nfreq=1000, dfreq=0.01, delta=0, epsilon=0.05, kk=1),
        # plasmon dispersion of silicon along a q line, only eps_M and the loss come back
        dict(name="line_si_plasmon", kind="line", crystal="si", switch="epsLL", precision="fp64", encut=110, n1=6,
             n2=6, n3=6, nq=6, neps=27, nband=24, nvalence=8, nfreq=1501, dfreq=0.02, delta=0, epsilon=0.1, kk=1),
        # screening of a set of crystals: uneven sizes, merged launches, eps_M only
        dict(name="batch_crystals", kind="batch", count=8, shape=11, precision="fp64", grid=4, nq=2, nfreq=1000,
             dfreq=0.025, delta=0, epsilon=0.1, kk=1),
        # one step of the parameter fit of tellurium: bands and eps_M, forward and backward
        dict(name="fit_te_step", kind="fit", crystal="te", switch="epsLL", precision="fp64", encut=120, points=40,
             n1=4, n2=4, n3=3, nq=1, neps=15, nband=24, nvalence=18, nfreq=1000, dfreq=0.01, delta=0, epsilon=0.05,
             kk=1),
        # post-processing of a saved spectrum (27 local-field vectors, 2000 frequencies) on host arrays
        dict(name="post_spectrum", kind="post", nq=1, neps=27, nfreq=2000, dfreq=0.0125),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["band", "chi", "chi", "chi", "chi", "line", "batch", "fit", "post"])
    if kind == "post":
        return dict(kind="post", nq=rng.randint(1, 3), neps=rng.choice([1, 9, 15, 20, 27, 33]),
                    nfreq=_log(rng, 150, 3001), dfreq=rng.choice([0.01, 0.0125, 0.02]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 7), shape=rng.randint(100, 999),
                    precision="fp64", grid=rng.randint(2, 4), nq=rng.randint(1, 2),
                    nfreq=_log(rng, 200, 1200), dfreq=0.025, delta=rng.choice([0, 0, 1, 2]), epsilon=0.1, kk=1)
    crystal = rng.choice(["si", "gaas", "wz", "te"])
    soc = crystal in ("gaas", "te")
    nvalence = {"si": 8, "gaas": 8, "wz": 16, "te": 18}[crystal]
    nband = nvalence + 2 * rng.randint(2, 10)
    encut = {"si": rng.randint(60, 220), "gaas": rng.randint(60, 180), "wz": rng.randint(110, 260),
             "te": rng.randint(50, 120)}[crystal]
    if kind == "band":
        return dict(kind="band", crystal=crystal, encut=encut, points=_log(rng, 8, 240), nband=nband,
                    nvalence=nvalence)
    if kind == "fit":
        return dict(kind="fit", crystal=crystal, switch="epsLL", precision="fp64", encut=min(encut, 110),
                    points=rng.randint(8, 30), n1=rng.randint(2, 3), n2=rng.randint(2, 3), n3=rng.randint(1, 3), nq=1,
                    neps=rng.choice([1, 9, 11, 15]), nband=nband, nvalence=nvalence, nfreq=_log(rng, 100, 1000),
                    dfreq=0.02, delta=rng.choice([0, 1]), epsilon=0.1, kk=1)
    case = dict(kind=kind, crystal=crystal, switch="epsLL" if kind == "line" else rng.choice(["epsLL", "epsij"]),
                precision="fp64" if kind == "line" else rng.choice(["fp64", "mixed"]), encut=encut, n1=_log(rng, 2, 7), n2=_log(rng, 2, 7),
                n3=_log(rng, 1, 6), nq=rng.randint(2, 4) if kind == "line" else rng.choice([1, 1, 2]),
                neps=rng.choice([1, 9, 15, 20, 27, 33, 51] if not soc else [1, 9, 15, 20, 27]), nband=nband,
                nvalence=nvalence, nfreq=_log(rng, 200, 2500), dfreq=rng.choice([0.01, 0.0125, 0.02]),
                delta=rng.choice([0, 0, 1, 2, 3]), epsilon=rng.choice([0.05, 0.1]), kk=1)
    if case["switch"] == "epsij":
        case["kk"] = rng.choice([0, 1, 1])
    return case


# ------------------------------------------------------------------ crystals
class _Lattice:
    """Reciprocal basis, atoms and zone volume of a preset (units 2 pi / a, a)."""

    def __init__(self, preset, a, f=None, u=None):
        self.preset, self.a, self.f, self.u = preset, a, f, u
        s3 = math.sqrt(3.0)
        if preset in ("zb", "rs"):
            self.b = np.array([[-1, 1, 1], [1, -1, 1], [1, 1, -1]], float)
            self.tau = np.array([[0, 0, 0], [0.25] * 3 if preset == "zb" else [0.5, 0, 0]], float)
            self.volume = 4.0
        else:
            self.b = np.array([[1, -1 / s3, 0], [1, 1 / s3, 0], [0, 0, 1.0 / f]])
            self.volume = abs(np.linalg.det(self.b))
            if preset == "wz":
                self.tau = np.array([[0.5, 0.5 / s3, 0], [0.5, -0.5 / s3, 0.5 * f], [0.5, 0.5 / s3, u * f],
                                     [0.5, -0.5 / s3, (0.5 + u) * f]])
            else:
                self.tau = np.array([[0, 0.5 * s3 * u, -f / 3.0], [1.5 * u, 0, 0], [0, -0.5 * s3 * u, f / 3.0]])

    def gvectors(self, encut):
        """(G, hkl) within the cutoff by length."""
        gcut = math.sqrt(encut * (self.a / (2 * math.pi)) ** 2 / KCON)
        r = np.arange(-math.ceil(gcut), math.ceil(gcut) + 1)
        hkl = np.array(np.meshgrid(r, r, r, indexing="ij")).reshape(3, -1).T
        length = np.linalg.norm(hkl @ self.b, axis=1)
        keep = length <= gcut + 1e-6
        order = np.argsort(length[keep], kind="stable")
        hkl = hkl[keep][order]
        return hkl @ self.b, hkl

    def args(self):
        out = ["-crystal", self.preset, "-a", repr(self.a)]
        return out + (["-f", repr(self.f), "-u", repr(self.u)] if self.f else [])


def _join(values):
    return ",".join(repr(float(v)) for v in values)


def _material(crystal, rng):
    """Shells, per-atom form factors [atom][shell] and spin-orbit parameters
    (lambda_S, lambda_A, shells of lambda_A) in Ry; rng moves them by a few per cent."""
    soc = None
    if crystal == "si":
        g2, v = [3.0, 4.0, 8.0, 11.0], np.array([[-0.21, 0, 0.04, 0.08]] * 2)
    elif crystal == "gaas":
        text, opts = wl.gaas_form_factors()
        x = np.array([float(t) for t in text.split(",")])
        g2, v = list(x[:4]), x[4:].reshape(2, 4)
        soc = [float(opts[2]), np.array([float(t.split(":")[1]) for t in opts[4].split(",")]), 4]
    elif crystal == "wz":
        x = np.array([float(t) for t in wl.wz_form_factors().split(",")])
        g2, v = list(x[:5]), x[5:].reshape(4, 5)
    else:
        th = wl.te_params()
        g2, v = [float("%.6f" % t) for t in wl.te_shells()], np.array([th[:8]] * 3)
        soc = [th[8], np.full(4, th[9]), 4]
    # atoms of one species move together
    groups = {"wz": [(0, 1), (2, 3)], "te": [(0, 1, 2)], "si": [(0, 1)]}.get(crystal, [(0,), (1,)])
    v = v.copy()
    for grp in groups:
        v[list(grp)] *= 1.0 + rng.uniform(-0.02, 0.02, v.shape[1])
    if soc:
        soc = [float(soc[0] * (1.0 + rng.uniform(-0.05, 0.05))), soc[1] * (1.0 + rng.uniform(-0.05, 0.05)), soc[2]]
    return g2, v, soc


def _material_args(g2, v, soc):
    out = ["-vg", _join(g2) + "," + _join(v.ravel())]
    if soc:
        out += ["-use_uniform_us_so", "-uniform_us_so_val", repr(soc[0]), "-ua_so",
                ",".join("%r:%r" % (float(k), float(x)) for k, x in zip(g2[:soc[2]], soc[1]))]
    return out


def _kgrid(lat, n, rng):
    """Uniform grid shifted off the symmetry points: k [N, 3]."""
    shift = rng.uniform(0.15, 0.35, 3)
    i3, i2, i1 = (x.ravel() for x in np.meshgrid(*(np.arange(m) for m in n[::-1]), indexing="ij"))
    x = (np.stack([i1, i2, i3], 1) + shift) / np.array(n)
    x -= np.round(x)
    return x @ lat.b


def _qlist(case, rng):
    q = np.array([[0.01, 0, 0]]) if case["nq"] == 1 else np.outer(np.linspace(0.05, 0.5, case["nq"]), [1.0, 0, 0])
    return q + rng.uniform(0, 0.002, 3)


class _Model:
    """Everything a case's crystal is defined by, from the case and the seed."""

    def __init__(self, case, seed):
        rng = np.random.default_rng([2024, int(seed)])
        self.lat = _Lattice(*CRYSTALS[case["crystal"]])
        self.g2, self.v, self.soc = _material(case["crystal"], rng)
        if "n1" in case:
            self.k = _kgrid(self.lat, (case["n1"], case["n2"], case["n3"]), rng)
            self.q = _qlist(case, rng)
        self.fit_move = rng.uniform(-1, 1, 64)

    def base_args(self, case):
        return (self.lat.args() + _material_args(self.g2, self.v, self.soc) +
                ["-encut", str(case["encut"]), "-nband", str(case["nband"]), "-nvalence", str(case["nvalence"])])


def _path_args(case):
    preset = CRYSTALS[case["crystal"]][0]
    seg = max(1, case["points"] // 4)
    return ["-switch", "band", "-qpath", PATHS[preset], "-qnum", ",".join([str(seg)] * 4)]


def _chi_args(case, q, k, switch):
    fd, path = tempfile.mkstemp(suffix=".txt")
    os.close(fd)
    pm.write_kfile(path, k, np.ones(len(k)))
    args = ["-switch", switch, "-kpoint", "0", "-kpointfile", path, "-qvec", _join(q.ravel()), "-neps",
            str(case["neps"]), "-nfreq", str(case["nfreq"]), "-dfreq", repr(case["dfreq"]), "-delta",
            str(case["delta"]), "-epsilon", repr(case["epsilon"]), "-kk", str(case["kk"])]
    return args, path


def _chi_problem(base, case, q, k, switch):
    args, path = _chi_args(case, q, k, switch)
    try:
        return pm.Problem(base + args)
    finally:
        os.unlink(path)


def _batch_shapes(case):
    """The crystals of a batch (structure, size, spin-orbit coupling, form
    factors), from the case alone."""
    r = np.random.default_rng([77, case["shape"]])
    out = []
    for _ in range(case["count"]):
        preset = ("zb", "rs", "wz")[r.integers(3)]
        lat = _Lattice(preset, round(float(r.uniform(4, 6.5)), 3), *((1.63, 0.375) if preset == "wz" else ()))
        target = int(r.integers(50, 300))
        encut = 40
        while len(lat.gvectors(encut)[0]) < target:
            encut += 10
        length2 = np.unique(np.round((lat.gvectors(200)[0] ** 2).sum(1), 6))
        g2 = [3.0, 4.0, 8.0, 11.0] if preset != "wz" else [float(x) for x in length2[1:6]]
        v = r.uniform(-0.3, 0.3, (2, len(g2)))
        v = v if preset != "wz" else v[[0, 0, 1, 1]]
        soc = [float(r.uniform(0.002, 0.01)), r.uniform(0, 0.005, 3), 3] if r.uniform() < 0.5 else None
        out.append(dict(lat=lat, encut=encut, g2=g2, v=v, soc=soc, neps=int(r.choice([15, 27])), nband=24,
                        nvalence=8 if preset != "wz" else 16))
    return out


# ------------------------------------------------------------------ prepare / run
_shared = {}


def _context():
    if "ctx" not in _shared:
        _shared["ctx"] = pm.Context(0)
    return _shared["ctx"]


def _switch(name):
    return {"epsLL": pm.SWITCH_EPSLL, "epsij": pm.SWITCH_EPSIJ}[name]


def _precision(case):
    return pm.PREC_MIXED if case["precision"] == "mixed" else pm.PREC_FP64


def prepare(case, seed):
    s = {"case": case, "ctx": _context()}
    kind = case["kind"]
    if kind == "post":
        s["re"], s["im"] = _saved_spectrum(case, seed)
        return s
    if kind == "batch":
        s["problems"] = []
        rng = np.random.default_rng([78, int(seed)])
        for c in _batch_shapes(case):
            v = c["v"] * (1.0 + rng.uniform(-0.02, 0.02, c["v"].shape[1]))
            k = _kgrid(c["lat"], (case["grid"],) * 3, rng)
            base = (c["lat"].args() + _material_args(c["g2"], v, c["soc"]) +
                    ["-encut", str(c["encut"]), "-nband", str(c["nband"]), "-nvalence", str(c["nvalence"])])
            s["problems"].append(_chi_problem(base, dict(case, neps=c["neps"]), _qlist(case, rng), k, "epsLL"))
        return s
    m = _Model(case, seed)
    base = m.base_args(case)
    if kind in ("band", "fit"):
        s["band"] = pm.Problem(base + _path_args(case))
    if kind != "band":
        s["problem"] = _chi_problem(base, case, m.q, m.k, case["switch"])
    if kind == "chi":
        info = s["problem"].info
        s["re"] = torch.empty(info.chi_values, dtype=torch.float64, device=_DEV)
        s["im"] = torch.empty_like(s["re"])
        s["eps"] = torch.empty((info.nq, info.nfreq), dtype=torch.complex128, device=_DEV)
    if kind == "fit":
        theta = s["band"].params()
        s["theta"] = torch.tensor(theta, dtype=torch.float64)
        star = torch.tensor(theta * (1.0 + 0.02 * m.fit_move[:len(theta)]), dtype=torch.float64)
        with torch.no_grad():
            s["E_star"] = pmad.band(star, s["band"], s["ctx"]).clone()
            s["t_star"] = pmad.eps_m(star, s["problem"], s["ctx"]).imag.clone()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "band":
        return {"E": ctx.band(s["band"])}
    if kind == "chi":
        ctx.chi_device(s["problem"], _switch(case["switch"]), _precision(case), s["re"].data_ptr(),
                       s["im"].data_ptr(), s["eps"].data_ptr())
        out = {"re": s["re"], "im": s["im"], "eps": s["eps"]}
        if case["precision"] == "mixed":
            out = {"re": out["re"].to(MIXED_TYPES[0]), "im": out["im"].to(MIXED_TYPES[0]),
                   "eps": out["eps"].to(MIXED_TYPES[1])}
        return out
    if kind == "line":
        _, _, eps = ctx.chi_epsm(s["problem"], _switch(case["switch"]), _precision(case), chi=False)
        loss, peak = ctx.eels(eps, case["dfreq"], 2.0)
        return {"eps": eps, "loss": loss, "peak": peak}
    if kind == "batch":
        res = ctx.chi_batch(s["problems"], pm.SWITCH_EPSLL, _precision(case), epsm=True, chi=False)
        return {"eps": [r[2] for r in res]}
    if kind == "fit":
        theta = s["theta"].clone().requires_grad_(True)
        E = pmad.band(theta, s["band"], ctx)
        eps = pmad.eps_m(theta, s["problem"], ctx)
        loss = ((E - s["E_star"]) ** 2).sum() + ((eps.imag - s["t_star"]) ** 2).sum()
        loss.backward()
        return {"loss": loss.detach(), "E": E.detach(), "eps": eps.detach(), "grad": theta.grad}
    nq, npair, nf = s["re"].shape
    re, im = ctx.kk(s["re"].reshape(-1, nf), s["im"].reshape(-1, nf), case["dfreq"])
    re, im = re.reshape(nq, npair, nf), im.reshape(nq, npair, nf)
    eps = ctx.eps_macroscopic(case["neps"], re, im)
    loss, peak = ctx.eels(eps, case["dfreq"], 1.0)
    return {"re": re, "im": im, "eps": eps, "loss": loss, "peak": peak}


def _saved_spectrum(case, seed):
    """A density-response block as a run without Kramers-Kronig leaves it:
    transitions with overlaps that fall off with |q + G|, Gaussian lines."""
    g = torch.Generator().manual_seed(int(seed))
    nq, neps, nf, nt = case["nq"], case["neps"], case["nfreq"], 96
    top = case["dfreq"] * nf
    m = torch.randn(nq, nt, neps, 2, generator=g, dtype=torch.float64)
    m = torch.view_as_complex(m) / (1.0 + torch.arange(neps, dtype=torch.float64)) ** 0.75
    e = 0.1 * top + 0.5 * top * torch.rand(nq, nt, generator=g, dtype=torch.float64)
    w = torch.arange(nf, dtype=torch.float64) * case["dfreq"]
    line = torch.exp(-0.5 * ((e[..., None] - w) / (0.01 * top)) ** 2)
    i, j = np.tril_indices(neps)
    o = (m[:, :, i] * m[:, :, j].conj()).transpose(1, 2)
    im = 0.2 * (o.real @ line)
    re = -0.2 * (o.imag @ line)
    return re.numpy(), im.numpy()


# ------------------------------------------------------------------ work
def _solve_work(n, m, count):
    """(bytes, flops) of `count` Hermitian eigenproblems of size n with m eigenvectors."""
    return 16.0 * n * m * count, (16.0 / 3.0 * n ** 3 + 8.0 * n * n * m) * count


def _chi_work(npw, soc, nk, nq, neps, nband, nvalence, nf, switch, delta, epsilon, dfreq, kk, whole):
    n, m = (2 * npw, nband) if soc else (npw, nband // 2)
    nb, nf_ = _solve_work(n, m, nk * (1 + nq))
    nv = nvalence if soc else nvalence // 2
    trans = nk * nq * nv * (m - nv)
    npair = neps * (neps + 1) // 2
    width = nf
    if switch == "epsij":
        width = min(nf, 2 * max(1, int((50 if delta == 1 else 6) * epsilon / dfreq)) + 1)
    elif delta == 0:
        width = min(nf, 2 * int(38.7 * epsilon / dfreq) + 1)  # beyond, the Gaussian is zero in FP64
    elif delta >= 2:
        width = min(nf, int(epsilon / dfreq) + 1)
    blocks = 9 if whole else 1
    channels = 10 if soc and switch == "epsij" else 4
    flops = nf_ + 8.0 * channels * trans * neps * npw + 4.0 * blocks * npair * trans * width
    out = 16.0 * blocks * npair * nf * nq
    if kk:
        flops += 4.0 * 5.0 * 2 * nf * math.log2(2.0 * nf + 2) * blocks * npair * nq
    flops += 8.0 / 3.0 * neps ** 3 * nf * nq
    return nb + out + 16.0 * nf * nq, flops


def work(case):
    kind = case["kind"]
    if kind == "post":
        rows = case["nq"] * case["neps"] * (case["neps"] + 1) // 2
        nf = case["nfreq"]
        return {"bytes": 4.0 * 8 * rows * nf + 40.0 * case["nq"] * nf,
                "flops": 4.0 * 5 * 2 * nf * math.log2(2.0 * nf + 2) * rows +
                8.0 / 3.0 * case["neps"] ** 3 * nf * case["nq"]}
    if kind == "batch":
        b = f = 0.0
        for c in _batch_shapes(case):
            npw = len(c["lat"].gvectors(c["encut"])[0])
            x, y = _chi_work(npw, c["soc"], case["grid"] ** 3, case["nq"], c["neps"], c["nband"], c["nvalence"],
                             case["nfreq"], "epsLL", case["delta"], case["epsilon"], case["dfreq"], case["kk"], False)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    lat = _Lattice(*CRYSTALS[case["crystal"]])
    npw = len(lat.gvectors(case["encut"])[0])
    soc = case["crystal"] in ("gaas", "te")
    n = 2 * npw if soc else npw
    b = f = 0.0
    if kind in ("band", "fit"):
        b, f = _solve_work(n, 0, 4 * max(1, case["points"] // 4) + 2)
        b += 8.0 * case["points"] * case["nband"]
    if kind != "band":
        x, y = _chi_work(npw, soc, case["n1"] * case["n2"] * case["n3"], case["nq"], case["neps"], case["nband"],
                         case["nvalence"], case["nfreq"], case["switch"], case["delta"], case["epsilon"],
                         case["dfreq"], case["kk"], kind == "chi")
        b, f = b + x, f + y
    if kind == "fit":  # the adjoint needs the eigenpairs again and as many products with each H
        b, f = 2 * b, 2 * f
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact values
def _hamiltonians(lat, g2, v, soc, G, hkl, k):
    """H(k) [len(k), n, n] of the plane-wave basis (spinor with spin-orbit coupling)."""
    dev = _DEV
    npw = len(G)
    d = hkl[:, None, :] - hkl[None, :, :]
    dG = d @ lat.b
    len2 = (dG ** 2).sum(-1)
    phase = dG @ lat.tau.T
    pot = np.zeros((npw, npw), complex)
    for s, key in enumerate(g2):
        shell = (abs(len2 - key) < 1e-2) & (len2 < g2[-1] + 1e-2)
        pot[shell] = (np.exp(-2j * np.pi * phase[shell]) * v[:, s]).mean(-1) * RY
    np.fill_diagonal(pot, 0.0)
    pot = torch.tensor(pot, device=dev)
    kg = torch.tensor(G[None] + k[:, None], device=dev)
    kin = KCON * (2 * math.pi / lat.a) ** 2
    h0 = pot + torch.diag_embed((kin * (kg ** 2).sum(-1)).to(torch.complex128))
    if not soc:
        return h0
    vso = np.where(len2 > 1e-9, 1.0, 0.0) * soc[0] * RY * np.cos(2 * np.pi * -phase).mean(-1) + 0j
    for key, x in zip(g2[:soc[2]], soc[1]):
        shell = abs(len2 - key) < 1e-2
        vso[shell] += 1j * x * RY * np.sin(2 * np.pi * -phase[shell]).mean(-1)
    vso = torch.tensor(vso, device=dev)
    h = torch.zeros(len(k), npw, 2, npw, 2, dtype=torch.complex128, device=dev)
    c = [1j * vso * x for x in torch.unbind(torch.linalg.cross(kg[:, None, :, :].expand(-1, npw, -1, -1),
                                                              kg[:, :, None, :].expand(-1, -1, npw, -1)), -1)]
    h[:, :, 0, :, 0] = h0 + c[2]
    h[:, :, 1, :, 1] = h0 - c[2]
    h[:, :, 0, :, 1] = c[0] - 1j * c[1]
    h[:, :, 1, :, 0] = c[0] + 1j * c[1]
    low = torch.tril(h.reshape(len(k), 2 * npw, 2 * npw))
    return low + torch.tril(low, -1).conj().transpose(1, 2)


def _eigenpairs(lat, g2, v, soc, G, hkl, k, vectors):
    w, z = [], []
    for i in range(0, len(k), 32):
        h = _hamiltonians(lat, g2, v, soc, G, hkl, k[i:i + 32])
        if vectors:
            a, b = torch.linalg.eigh(h)
            z.append(b)
        else:
            a = torch.linalg.eigvalsh(h)
        w.append(a)
    return torch.cat(w), (torch.cat(z) if vectors else None)


def _reference_energy(lat, g2, v, soc, G, hkl, nvalence):
    w = _eigenpairs(lat, g2, v, soc, G, hkl, np.zeros((1, 3)), False)[0][0]
    w = w if soc else w.repeat_interleave(2)
    return float(w[nvalence - 1] + w[nvalence]) / 2


def _path_points(lat, points):
    s3, f = math.sqrt(3.0), lat.f
    if lat.preset == "zb":
        at = {"G": (0, 0, 0), "X": (1, 0, 0), "W": (1, 0.5, 0), "L": (0.5, 0.5, 0.5)}
    else:
        at = {"G": (0, 0, 0), "A": (0, 0, 0.5 / f), "H": (2 / 3, 0, 0.5 / f), "K": (2 / 3, 0, 0)}
    names = PATHS[lat.preset].split(",")
    seg = max(1, points // 4)
    out = [np.array(at[names[0]], float)]
    for x, y in zip(names, names[1:]):
        x, y = np.array(at[x], float), np.array(at[y], float)
        out += [x + (y - x) * (i / seg) for i in range(1, seg + 1)]
    return np.array(out)


def _bands(model, case):
    G, hkl = model.lat.gvectors(case["encut"])
    args = (model.lat, model.g2, model.v, model.soc, G, hkl)
    w = _eigenpairs(*args, _path_points(model.lat, case["points"]), False)[0]
    w = w if model.soc else w.repeat_interleave(2, dim=1)
    return w[:, :case["nband"]] - _reference_energy(*args, case["nvalence"])


def _line_shape(case, x):
    e = case["epsilon"]
    if case["delta"] == 0:
        return torch.exp(-0.5 * (x / e) ** 2) / (e * math.sqrt(2 * math.pi))
    if case["delta"] == 1:
        return e / math.pi / (e * e + x * x)
    inside = (x.abs() < 0.5 * e).to(x.dtype)
    return inside * (4 / e * (0.5 - x.abs() / e)) if case["delta"] == 2 else inside / e


def _polarisation(q):
    """Unit vector along q + G."""
    n = np.linalg.norm(q, axis=-1, keepdims=True)
    return q / n


def _eps(model, case):
    """eps_M [nq, nfreq] from the longitudinal block; None where the order of
    the local-field vectors is not known here."""
    lat, soc, neps = model.lat, model.soc, case["neps"]
    G, hkl = lat.gvectors(case["encut"])
    order = _ORDER.get((case["crystal"], case["encut"]), "0,0,0").split()
    if neps > len(order):
        return None
    first = [tuple(int(x) for x in t.split(",")) for t in order]
    hkl = np.array(first + [h for h in map(tuple, hkl) if h not in set(first)])
    G = hkl @ lat.b
    args = (lat, model.g2, model.v, soc, G, hkl)
    off = _reference_energy(*args, case["nvalence"])
    ns = case["nband"] if soc else case["nband"] // 2
    where = {tuple(h): i for i, h in enumerate(hkl)}
    loci = torch.tensor([[where.get(tuple(h + hkl[m]), -1) for h in hkl] for m in range(neps)], device=_DEV)
    sw = 2 if soc else 1
    nf, df = case["nfreq"], case["dfreq"]
    omega = torch.arange(nf, device=_DEV, dtype=torch.float64) * df
    i, j = np.tril_indices(neps)
    ij = case["switch"] == "epsij"
    acm = lat.a * 1e-8
    wk, zk = _eigenpairs(*args, model.k, True)
    wk, zk = wk[:, :ns] - off, zk[:, :, :ns].reshape(len(model.k), len(G), sw, ns)
    Gt = torch.tensor(G, device=_DEV)
    out = []
    for q in model.q:
        wq, zq = _eigenpairs(*args, model.k + q, True)
        wq, zq = wq[:, :ns] - off, zq[:, :, :ns].reshape(len(model.k), len(G), sw, ns)
        u = _polarisation(q + G[:neps])
        acc = [torch.zeros(len(i), nf, dtype=torch.float64, device=_DEV) for _ in range(2)]
        for k in range(len(model.k)):
            c, v = wk[k] > 0, wq[k] <= 0
            if not c.any() or not v.any():
                continue
            de = (wk[k][c][:, None] - wq[k][v][None]).reshape(-1)
            zc, zv = zk[k][:, :, c], zq[k][:, :, v]
            ch = []
            for m in range(neps):
                on = loci[m] >= 0
                a, b = zc[on].conj(), zv[loci[m][on]]
                if not ij:
                    ch.append(torch.einsum("psc,psv->cv", a, b).reshape(1, -1))
                    continue
                um = torch.tensor(u[m], device=_DEV)
                orb = (Gt[on] + torch.tensor(model.k[k] + q / 2 + G[m] / 2, device=_DEV)) @ um
                same = torch.einsum("psc,p,psv->scv", a, orb.to(a.dtype), b)
                if not soc:
                    ch.append(same.reshape(1, -1))
                    continue
                g2m = float((G[m] ** 2).sum())
                la = next((float(x) for key, x in zip(model.g2[:soc[2]], soc[1]) if abs(key - g2m) < 1e-2), 0.0)
                vso = 1j * la * RY * float(np.sin(2 * np.pi * (lat.tau @ G[m])).mean())
                cur = 1j * vso * np.array([G[m][1] + 1j * G[m][2], G[m][2] - G[m][0], -1j * G[m][0] - G[m][1]])
                s = complex(u[m] @ cur)
                ud = s * torch.einsum("pc,pv->cv", a[:, 0], b[:, 1])
                du = s * torch.einsum("pc,pv->cv", a[:, 1], b[:, 0])
                ch.append(torch.stack([same[0], same[1], ud, du]).reshape(4, -1))
            M = torch.stack(ch)                                     # [neps, channel, transition]
            A, B = M[i], M[j].conj()
            if M.shape[1] == 1:
                o = (A * B)[:, 0]
                re_o, im_o = o.real, o.imag
            else:
                t = A[:, 0] * B[:, 0] + A[:, 1] * B[:, 1] - A[:, 2] * B[:, 2] - A[:, 3] * B[:, 3]
                x = A[:, 0] * B[:, 1] + A[:, 1] * B[:, 0] - A[:, 3] * B[:, 2] - A[:, 2] * B[:, 3]
                re_o, im_o = t.real + x.real, t.imag
            weight = (1.0 if soc else 2.0) / len(model.k)
            shape = _line_shape(case, de[:, None] - omega)
            if ij:
                half = max(1, int((50 if case["delta"] == 1 else 6) * case["epsilon"] / df))
                f0 = torch.trunc(de / df)
                shape = shape * ((torch.arange(nf, device=_DEV) - f0[:, None]).abs() <= half)
            acc[0] -= weight * (im_o @ shape)
            acc[1] += weight * (re_o @ shape)
        if ij:
            sf = (4.0 * lat.volume * math.pi ** 5 * HBAR ** 4 * ESU ** 2 / (EV ** 3 * EM ** 2 * acm ** 5))
            inv = torch.where(omega > 0, 1.0 / torch.where(omega > 0, omega, 1.0) ** 2, 0.0)
            chi = [sf * x * inv for x in acc]
        else:
            n = np.linalg.norm(q + G[:neps], axis=1)
            sf = torch.tensor(2.0 * lat.volume * ESU ** 2 / (math.pi * EV * acm) / (n[i] * n[j]), device=_DEV)
            chi = [math.pi * x * sf[:, None] * (omega > 0) for x in acc]
        if case["kk"]:
            chi = _kramers_kronig(chi[0], chi[1], omega, df)
        out.append(_macroscopic(chi[0], chi[1], neps))
    return torch.stack(out)


def _kramers_kronig(re, im, omega, df):
    den = omega[None, :] ** 2 - omega[:, None] ** 2
    kern = torch.where(den == 0, 0.0, omega[None, :] / torch.where(den == 0, 1.0, den)).T * (2 * df / math.pi)
    return [re + im @ kern, im + re @ kern]


def _macroscopic(re, im, neps):
    i, j = np.tril_indices(neps)
    e = torch.zeros(re.shape[-1], neps, neps, dtype=torch.complex128, device=re.device)
    z = torch.complex(re, im).T
    e[:, j, i] = z.conj()
    e[:, i, j] = z
    e = e + torch.eye(neps, dtype=torch.complex128, device=re.device)
    return 1.0 / torch.linalg.inv(e)[:, 0, 0]


def _loss(eps, df, wmin):
    loss = -(1.0 / eps).imag
    first = max(0, math.ceil(wmin / df - 1e-9))
    peaks = []
    for row in loss.cpu().numpy():
        p = first + int(np.argmax(row[first:]))
        at, top = p * df, row[p]
        if 0 < p < len(row) - 1:
            a, b, c = row[p - 1], row[p], row[p + 1]
            if a - 2 * b + c < 0:
                t = 0.5 * (a - c) / (a - 2 * b + c)
                at, top = (p + t) * df, b - 0.25 * (a - c) * t
        peaks.append((at, top))
    return loss, np.array(peaks)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    if kind == "post":
        re, im = (torch.tensor(x, device=_DEV) for x in _saved_spectrum(case, seed))
        omega = torch.arange(case["nfreq"], device=_DEV, dtype=torch.float64) * case["dfreq"]
        re, im = _kramers_kronig(re, im, omega, case["dfreq"])
        eps = torch.stack([_macroscopic(r, i, case["neps"]) for r, i in zip(re, im)])
        loss, peak = _loss(eps, case["dfreq"], 1.0)
        return {"re": re, "im": im, "eps": eps, "loss": loss, "peak": peak}
    m = _Model(case, seed)
    soc = case["crystal"] in ("gaas", "te")
    n = len(m.lat.gvectors(case["encut"])[0]) * (2 if soc else 1)
    solves = (case["points"] if kind == "band" else len(m.k) * (1 + case["nq"]))
    if solves * (n / 100.0) ** 2 > 9000:  # about 20 seconds of one-by-one eigenproblems
        return None
    if kind == "band":
        return {"E": _bands(m, case)}
    eps = _eps(m, case)
    if kind == "chi":
        return {"re": None, "im": None, "eps": eps} if eps is not None else None
    if kind == "line":
        loss, peak = _loss(eps, case["dfreq"], 2.0) if eps is not None else (None, None)
        return {"eps": eps, "loss": loss, "peak": peak} if eps is not None else None
    return {"loss": None, "E": _bands(m, case), "eps": eps, "grad": None}
