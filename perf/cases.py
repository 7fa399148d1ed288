"""Timed cases: what a user of this framework has it compute, through its public entry points.

A case names a kind of call and its sizes:

  curve     ProfileCalculator.calculate, the default way to a scattering curve (method Auto: Debye sums below 500
            atoms, else the multipole expansion), with and without a hydration shell
  debye     debye_solvent_basis, the six Debye terms that every (c1, c2) recombines
  gradient  chi2_grad, chi squared of a curve and its gradient in every coordinate (forward and backward)
  fit       SaxsScorer.score, a structure fitted to a measured curve
  ensemble  EnsemblePlan.score, conformers weighted against a measured curve
  pr        coordinate_features, the pair-distance distribution
  grids     both hydration grids

Structures are seeded globules of the density of a protein with coordinates to 0.001 Angstrom, as coordinate files
hold them.  "united" gives their atoms the united-atom groups of a real residue list (a dozen scattering classes
instead of four), "altloc" gives one atom in 25 a partial occupancy to two decimals, and "measured" takes a q grid as
a data file has it (q to five decimals, so the steps are not quite equal).

Curves, gradients and fits are summed in single precision (FP32 pair sums, TF32 hi + lo moments), so they are returned
in that type; grids, P(r) and site lists are exact in double precision and are returned as such.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import crabsaxs_b200 as cs

C, N_, O_, S_ = 1, 2, 3, 4  # element codes of the four elements below
DENSITY = 0.334  # electrons per cubic Angstrom of bulk water


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a peptide's curve in vacuum, latency only
        dict(name="curve_300", kind="curve", atoms=300, nq=101, qmax=0.5, hydration="none", united=True),
        # a small protein with its hydration grid at the default settings
        dict(name="curve_1481_grid4", kind="curve", atoms=1481, nq=101, qmax=0.5, hydration="adaptive", spacing=4.0,
             united=True),
        # a large complex, the same settings
        dict(name="curve_58870_grid4", kind="curve", atoms=58870, nq=101, qmax=0.5, hydration="adaptive", spacing=4.0,
             united=True),
        # the largest curve: 100,000 atoms, 1000 q, order 50
        dict(name="curve_100000_l50", kind="curve", atoms=100000, nq=1000, qmax=0.6, hydration="none", l_max=50),
        # exact Debye terms: a small protein, a ragged one with partial occupancies on a measured grid, and a large
        # one with its hydration sites
        dict(name="debye_1000", kind="debye", atoms=1000, nq=100, qmax=0.5, hydration="analytic", united=True),
        dict(name="debye_7321_measured", kind="debye", atoms=7321, nq=333, qmax=0.45, hydration="analytic",
             united=True, altloc=True, measured=True),
        dict(name="debye_20000_grid3", kind="debye", atoms=20000, nq=500, qmax=0.5, hydration="adaptive",
             spacing=3.0),
        # one step of a refinement against data
        dict(name="gradient_5000", kind="gradient", atoms=5000, nq=100, qmax=0.5),
        # a fit of scale, background, c1 and c2 to a measured curve
        dict(name="fit_1481", kind="fit", atoms=1481, nq=612, qmax=0.5, spacing=8.0, united=True, measured=True),
        # conformers of different sizes scored against one curve
        dict(name="ensemble_48", kind="ensemble", conformers=48, atoms=2000, most=16000, nq=300, qmax=0.45),
        # pair-distance distribution of the largest structure
        dict(name="pr_100000", kind="pr", atoms=100000, bins=160),
        # hydration grids alone
        dict(name="grids_20000", kind="grids", atoms=20000, spacing=3.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["curve", "curve", "debye", "debye", "debye", "gradient", "fit", "ensemble", "pr", "grids"])
    united = rng.random() < 0.6
    altloc = rng.random() < 0.3
    qmax = round(rng.uniform(0.3, 0.6), 3)
    if kind == "curve":
        case = dict(kind=kind, atoms=_log(rng, 200, 100000), nq=_log(rng, 50, 1000), qmax=qmax,
                    hydration=rng.choice(["none", "analytic", "adaptive", "adaptive"]),
                    spacing=rng.choice([3.0, 4.0, 8.0]))
    elif kind == "debye":
        case = dict(kind=kind, atoms=_log(rng, 100, 20000), nq=_log(rng, 50, 500), qmax=min(qmax, 0.5),
                    hydration=rng.choice(["analytic", "analytic", "adaptive"]), spacing=rng.choice([3.0, 4.0, 8.0]))
        case["measured"] = case["atoms"] <= 7000 and case["nq"] <= 333 and rng.random() < 0.5
    elif kind == "gradient":
        case = dict(kind=kind, atoms=_log(rng, 200, 10000), nq=_log(rng, 50, 300), qmax=qmax)
    elif kind == "fit":
        case = dict(kind=kind, atoms=_log(rng, 500, 20000), nq=_log(rng, 100, 1000), qmax=qmax,
                    spacing=rng.choice([4.0, 8.0]), measured=True)
    elif kind == "ensemble":
        atoms = _log(rng, 500, 3000)
        return dict(kind=kind, conformers=_log(rng, 4, 48), atoms=atoms, most=atoms * rng.choice([1, 2, 4]),
                    nq=_log(rng, 50, 300), qmax=min(qmax, 0.45), united=united, altloc=False)
    elif kind == "pr":
        case = dict(kind=kind, atoms=_log(rng, 300, 100000), bins=_log(rng, 32, 500))
    else:
        case = dict(kind=kind, atoms=_log(rng, 300, 30000), spacing=rng.choice([3.0, 4.0, 8.0]))
    return dict(case, united=united, altloc=altloc)


# ------------------------------------------------------------------ inputs
def _globule(rng, n, united=False, altloc=False):
    """n atoms of a jittered lattice inside an ellipsoid, 19 cubic Angstrom each: (xyz, element, occupancy, group)."""
    axes = np.array([1.0, rng.uniform(0.7, 1.0), rng.uniform(0.5, 0.9)])
    axes /= axes.prod() ** (1.0 / 3.0)
    axes *= (19.0 * n * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
    a = 19.0 ** (1.0 / 3.0)
    ranges = [np.arange(-int(r / a) - 2, int(r / a) + 3) * a for r in axes]
    p = np.stack(np.meshgrid(*ranges, indexing="ij"), axis=-1).reshape(-1, 3)
    p = p + rng.normal(scale=0.4 * a, size=p.shape)
    inside = np.argsort(((p / axes) ** 2).sum(axis=1), kind="stable")[:n]
    xyz = np.round(p[rng.permutation(inside)] + rng.uniform(-30.0, 30.0, size=3), 3)
    element = rng.choice([C, N_, O_, S_], size=n, p=[0.63, 0.17, 0.19, 0.01]).astype(np.int8)
    group = np.full(n, -1, dtype=np.int8)
    if united:
        for e, groups, share in ((C, [-1, 0, 1, 2, 3], [0.30, 0.24, 0.24, 0.12, 0.10]),
                                 (N_, [-1, 7, 8, 10, 12], [0.05, 0.75, 0.06, 0.06, 0.08]),
                                 (O_, [-1, 4, 6], [0.76, 0.10, 0.14]), (S_, [-1, 13], [0.6, 0.4])):
            at = element == e
            group[at] = rng.choice(groups, size=int(at.sum()), p=share)
    occupancy = np.ones(n)
    if altloc:
        at = rng.random(n) < 0.04
        occupancy[at] = np.round(rng.uniform(0.3, 0.7, size=int(at.sum())), 2)
    return xyz, element, occupancy, group


def _q(rng, case):
    q = np.linspace(0.005, case["qmax"], case["nq"])
    if case.get("measured"):
        q = np.round(q, 5)
    return q


def _measured(rng, q, radius, scale):
    """A smooth curve of a globule of that radius with 3 % noise, and its errors."""
    rg = math.sqrt(0.6) * radius
    y = scale * (np.exp(-(q * rg) ** 2 / 3.0) + 0.02 / (1.0 + (q * radius / 3.0) ** 4) + 0.001)
    sigma = 0.03 * y + 1e-4 * scale
    return y + sigma * rng.normal(size=len(q)), sigma


def _solvent(case):
    kind = case.get("hydration", "analytic")
    if kind == "none":
        return None
    model = {"analytic": cs.HydrationModel.Analytic, "adaptive": cs.HydrationModel.AdaptiveGrid}[kind]
    return dict(c1=1.01, c2=1.1, model=model, spacing=float(case.get("spacing", 4.0)))


def _params(s):
    return cs.SolventParams(c1=s["c1"], c2=s["c2"], hydration_model=s["model"],
                            hydration_grid_spacing_angstrom=s["spacing"])


def _inputs(case, seed):
    """Everything a case is made of, from the seed alone."""
    rng = np.random.default_rng([int(seed), 7])
    v = {}
    if case["kind"] == "ensemble":
        sizes = np.round(np.exp(rng.uniform(math.log(case["atoms"]), math.log(case["most"]),
                                            size=case["conformers"]))).astype(int)
        v["atoms"] = [_globule(rng, int(n), case.get("united"), case.get("altloc")) for n in sizes]
        radius = (19.0 * float(sizes.mean()) * 0.75 / math.pi) ** (1.0 / 3.0)
    elif case["kind"] == "grids":
        # the number of sites depends on the structure: one globule per case (coordinates in 1/1024 Angstrom, so that
        # moving it is exact), the seed moves it and orders its atoms
        xyz, element, occupancy, group = _globule(np.random.default_rng([case["atoms"], 11]), case["atoms"])
        order = rng.permutation(case["atoms"])
        xyz = np.round(xyz * 1024.0) / 1024.0 + rng.integers(-32768, 32768, size=3) / 1024.0
        v["atoms"] = xyz[order], element[order], occupancy, group
        radius = 0.0
    else:
        v["atoms"] = _globule(rng, case["atoms"], case.get("united"), case.get("altloc"))
        radius = (19.0 * case["atoms"] * 0.75 / math.pi) ** (1.0 / 3.0)
    if "nq" in case:
        v["q"] = _q(rng, case)
        v["y"], v["sigma"] = _measured(rng, v["q"], radius, 1.0)
    if case["kind"] == "gradient":  # the scale that takes the structure's I(0) to the measured curve's
        xyz, w, cls, amp = _points(dict(case, hydration="analytic"), dict(v, q=np.zeros(1)), False)
        v["scale"] = float(1.0 / ((w * _combined(amp, np.zeros(1), "analytic")[cls, 0]).sum() ** 2))
    return v


def prepare(case, seed):
    v = _inputs(case, seed)
    kind = case["kind"]
    state = dict(kind=kind, engine=cs.Engine.default(0), q=v.get("q"), y=v.get("y"), sigma=v.get("sigma"))
    if kind == "ensemble":
        state["plan"] = cs.EnsemblePlan([cs.Structure(*a) for a in v["atoms"]], v["q"],
                                        solvent=cs.SolventParams())
        return state
    state["structure"] = cs.Structure(*v["atoms"])
    s = _solvent(case)
    if kind == "curve":
        options = cs.ComputeOptions(multipole_l_max=case.get("l_max"), solvent=None if s is None else _params(s))
        state["calculator"] = cs.ProfileCalculator(v["q"], options)
    elif kind == "debye":
        state["solvent"] = _params(s)
    elif kind == "gradient":
        state["solvent"] = _params(s)
        state["scale"] = v["scale"]
    elif kind == "fit":
        fit = cs.FitOptions(solvent=cs.SolventParams(hydration_model=cs.HydrationModel.AdaptiveGrid))
        quality = cs.Quality.Fast if case["spacing"] == 8.0 else cs.Quality.Balanced
        state["scorer"] = cs.SaxsScorer(cs.ExperimentalCurve(v["q"], v["y"], v["sigma"]),
                                        cs.ScoreOptions(fit=fit, quality=quality))
    elif kind == "pr":
        state["options"] = cs.PrOptions(bins=case["bins"])
    else:
        state["spacing"] = case["spacing"]
    return state


def _single(x):
    return np.asarray(x, dtype=np.float32)


def run(state):
    kind = state["kind"]
    if kind == "curve":
        return {"intensity": _single(state["calculator"].calculate(state["structure"]).intensity)}
    if kind == "debye":
        return {"basis": _single(cs.debye_solvent_basis(state["structure"], state["q"], state["solvent"]))}
    if kind == "gradient":
        chi2, gx, gp = cs.chi2_grad(state["structure"], state["q"], state["y"], state["sigma"], state["solvent"],
                                    state["scale"], 0.0)
        return {"chi2": _single(chi2), "grad_xyz": _single(gx), "grad_params": _single(gp)}
    if kind == "fit":
        r = state["scorer"].score(state["structure"])
        p = r.fit.params
        return {"curve": _single(r.fit.fitted_curve), "chi2": _single(r.chi2),
                "params": _single([p.scale, p.background, p.c1, p.c2])}
    if kind == "ensemble":
        r = state["plan"].score(state["y"], state["sigma"])
        return {"candidate": r["candidate"], "weights": _single(r["weights"]), "dchi2_dw": _single(r["dchi2_dw"]),
                "fit": _single([r["c1"], r["c2"], r["scale"], r["background"], r["reduced_chi2"]]),
                "dchi2_dc": _single([r["dchi2_dc1"], r["dchi2_dc2"]]), "kl_weights": _single(r["kl_weights"]),
                "kl_chi2": _single(r["kl_reduced_chi2"])}
    if kind == "pr":
        f = cs.coordinate_features(state["structure"], state["options"])
        return {"rg": f.rg, "dmax": f.dmax, "r": f.p_r.r, "p": f.p_r.p}
    adaptive, va = cs.hydration_grid_adaptive(state["structure"], state["spacing"])
    exterior, ve = cs.hydration_grid_exterior(state["structure"])
    return {"adaptive": adaptive, "exterior": exterior, "volumes": [va, ve]}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: inputs once and outputs once.  Operations: ten per pair of points for a distance and its deposit; for an
    expansion, a multiply-add per harmonic and point and per harmonic and q."""
    kind, nq = case["kind"], case.get("nq", 0)
    if kind == "ensemble":
        lo, hi, k = case["atoms"], case["most"], case["conformers"]
        mean2 = lo * lo if hi == lo else (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        mean = lo if hi == lo else (hi - lo) / math.log(hi / lo)
        return {"bytes": k * mean * 34.0 + 24.0 * nq + 24.0 * k, "flops": 10.0 * k * mean2 / 2.0 + 50.0 * k * nq}
    n = case["atoms"]
    size = n * 34.0 + 16.0 * nq
    radius = (19.0 * n * 0.75 / math.pi) ** (1.0 / 3.0)
    sites = 0.0
    if kind != "pr" and (case.get("hydration") == "adaptive" or kind in ("fit", "grids")):
        sites = 4.0 * math.pi * (radius + 5.5) ** 2 * 5.0 / case["spacing"] ** 3
    if kind == "grids":
        outer = 4.0 * math.pi * (radius + 3.5) ** 2 * 4.0
        return {"bytes": size + 24.0 * (sites + outer), "flops": 10.0 * (n * 60.0 + (2.0 * radius + 10.0) ** 3)}
    if kind == "pr":
        return {"bytes": size + 16.0 * case["bins"], "flops": 10.0 * n * n / 2.0}
    points = n + sites
    if kind == "fit" or (kind == "curve" and n >= 500):
        order = case.get("l_max") or min(64.0, math.ceil(1.3 * case["qmax"] * radius) + 8.0)
        return {"bytes": size, "flops": 2.0 * (order + 1.0) ** 2 * (points + nq)}
    if kind == "gradient":
        return {"bytes": size + 24.0 * n, "flops": 10.0 * n * n / 2.0 + 20.0 * n * n / 2.0}
    return {"bytes": size + 48.0 * nq, "flops": 10.0 * points * points / 2.0}


# ------------------------------------------------------------------ the same in 64 bits
# Cromer-Mann coefficients (a1, b1, ..., a4, b4, c) of H, C, N, O, S and the five-Gaussian united-atom fits of
# Grudinin et al. 2017, with the displaced volumes of the elements and the hydrogens of each group
_ELEMENT = {
    0: ([0.493002, 0.322912, 0.140191, 0.04081], [10.5109, 26.1257, 3.14236, 57.7997], 0.003038),
    C: ([2.31, 1.02, 1.5886, 0.865], [20.8439, 10.2075, 0.5687, 51.6512], 0.2156),
    N_: ([12.2126, 3.1322, 2.0125, 1.1663], [0.0057, 9.8933, 28.9975, 0.5826], -11.529),
    O_: ([3.0485, 2.2868, 1.5463, 0.867], [13.2771, 5.7011, 0.3239, 32.9089], 0.2508),
    S_: ([6.9053, 5.2034, 1.4379, 1.5863], [1.4679, 22.2151, 0.2536, 56.172], 0.8669),
}
_GROUP = {
    0: ([2.909530, 0.485267, 1.516151, 0.206905, 1.541626], [13.933084, 23.221524, 41.990403, 4.974183, 0.679266],
        0.337670),
    1: ([3.275723, 0.870037, 1.534606, 0.395078, 1.544562], [13.408502, 23.785175, 41.922444, 5.019072, 0.724439],
        0.377096),
    2: ([3.681341, 1.228691, 1.549320, 0.574033, 1.554377], [13.026207, 24.131974, 41.869426, 4.984373, 0.765769],
        0.409294),
    3: ([2.168070, 1.275811, 1.561096, 0.742395, -6.151144], [12.642907, 18.420069, 41.768517, 1.535360, -0.045937],
        7.400917),
    4: ([0.456221, 3.219608, 0.812773, 2.666928, 1.380927], [21.503498, 13.397134, 34.547137, 5.826620, 0.412902],
        0.463202),
    6: ([0.688944, 2.929687, 0.416472, 2.606983, 1.319232], [29.319200, 6.572228, 64.951658, 16.267799, 0.455640],
        0.537548),
    7: ([1.650531, 0.429639, 2.144736, 1.851894, 1.408921], [10.603730, 6.987283, 29.939901, 10.573859, 0.611678],
        0.510589),
    8: ([1.904157, 1.942536, 2.435585, 0.730512, 1.379728], [10.803702, 10.792421, 29.610479, 6.847755, 0.709687],
        0.603738),
    10: ([1.882162, 1.933200, 2.465843, 0.927311, 1.190889], [10.975157, 10.956008, 29.208572, 6.663555, 0.843650],
         0.597322),
    12: ([1.792216, 0.724464, 2.347044, 1.903020, 1.313042], [10.830060, 6.846763, 29.579607, 10.800018, 0.720448],
         0.583312),
    13: ([0.570042, 6.337416, 1.641643, 5.398549, 1.527982], [11.447986, 1.197657, 55.401032, 22.420955, 2.356552],
         1.523944),
}
_GROUP_H = {0: 1, 1: 2, 2: 3, 3: 1, 4: 1, 6: 0, 7: 1, 8: 2, 10: 3, 12: 2, 13: 1}
_VOLUME = {0: 5.15, C: 16.44, N_: 2.49, O_: 9.13, S_: 26.09}


def _gauss(table, q):
    a, b, c = table
    s2 = (q / (4.0 * math.pi)) ** 2
    return sum(x * np.exp(-y * s2) for x, y in zip(a, b)) + c


def _classes(element, group):
    """The distinct (element, group) classes and each atom's class."""
    key = element.astype(np.int64) * 32 + group + 1
    keys, cls = np.unique(key, return_inverse=True)
    return [(int(k) // 32, int(k) % 32 - 1) for k in keys], cls.reshape(-1)


def _amplitudes(e, g, q, multipole):
    """Vacuum, displaced-solvent and analytic-shell amplitudes of a class."""
    v = _gauss(_GROUP[g] if g >= 0 else _ELEMENT[e], q)
    volume = _VOLUME[e] + (_GROUP_H[g] * _VOLUME[0] if g >= 0 else 0.0)
    ex = DENSITY * volume * np.exp(-(volume ** (2.0 / 3.0)) * q * q / (4.0 * math.pi))
    rs = (3.0 * volume / (4.0 * math.pi)) ** (1.0 / 3.0) + 1.5
    shell = 4.0 * math.pi * rs * rs * 3.0
    fall = rs * rs * q * q / 4.0 if multipole else shell ** (2.0 / 3.0) * q * q / (4.0 * math.pi)
    return v, ex, DENSITY * 0.1 * shell * np.exp(-fall)


def _water(q, spacing):
    """Amplitude of one grid site."""
    x = q * 0.9572
    f = _gauss(_ELEMENT[O_], q) + 2.0 * _gauss(_ELEMENT[0], q) * np.sin(x) / x
    volume = 2.0 * (spacing / 2.0) ** 3 if spacing > 4.0 else spacing ** 3
    return DENSITY / 10.0 * volume * f


def _shell_sites(xyz, spacing):
    """Voxels of the adaptive shell: beyond 3 Angstrom of every atom, within 3 plus the shell's width of one."""
    d = xyz - xyz.mean(axis=0)
    rg = math.sqrt((d * d).sum(axis=1).mean())
    outer = 3.0 + min(5.0, max(3.0, 3.0 + 0.4 * (rg - 15.0)))
    lo, hi = xyz.min(axis=0) - 12.0, xyz.max(axis=0) + 12.0
    dim = [int(math.ceil((hi[k] - lo[k]) / spacing - 1e-10)) + 1 for k in range(3)]
    masks = [np.zeros(dim, dtype=bool) for _ in range(2)]
    base = np.floor((xyz - lo) / spacing).astype(np.int64)
    reach = int(math.ceil(outer / spacing)) + 1
    for dx in range(-reach, reach + 1):
        for dy in range(-reach, reach + 1):
            for dz in range(-reach, reach + 1):
                cell = base + np.array([dx, dy, dz])
                ok = ((cell >= 0) & (cell < np.array(dim))).all(axis=1)
                cell = cell[ok]
                p = lo + cell * spacing - xyz[ok]
                d2 = p[:, 0] ** 2 + p[:, 1] ** 2 + p[:, 2] ** 2
                for mask, r in zip(masks, (outer, 3.0)):
                    near = cell[d2 <= r * r + 1e-10]
                    mask[near[:, 0], near[:, 1], near[:, 2]] = True
    at = np.argwhere((masks[0] & ~masks[1]).transpose(2, 1, 0))[:, ::-1]  # z, then y, then x
    return lo + at * spacing


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pair_sums(xyz, w, cls, n_cls, q):
    """S[a, b, k], the sum of w_i w_j sin(q r) / (q r) over i of class a and j of class b, itself included."""
    dev = _device()
    groups = [np.nonzero(cls == a)[0] for a in range(n_cls)]
    pts = [torch.tensor(xyz[g], dtype=torch.float64, device=dev) for g in groups]
    ws = [torch.tensor(w[g], dtype=torch.float64, device=dev) for g in groups]
    out = torch.zeros((n_cls, n_cls, len(q)), dtype=torch.float64, device=dev)
    for a in range(n_cls):
        for b in range(a, n_cls):
            if len(groups[a]) == 0 or len(groups[b]) == 0:
                continue
            rows = max(1, 6_000_000 // len(groups[b]))
            for i in range(0, len(groups[a]), rows):
                p = pts[a][i:i + rows]
                r2 = torch.zeros((p.shape[0], pts[b].shape[0]), dtype=torch.float64, device=dev)
                for d in range(3):
                    r2 += (p[:, d, None] - pts[b][None, :, d]) ** 2
                r = r2.sqrt_()
                zero = r < 1e-12
                ww = ws[a][i:i + rows, None] * ws[b][None, :]
                extra = (ww * zero).sum()
                ww = torch.where(zero, torch.zeros_like(ww), ww / r.clamp_min(1e-12))
                x = torch.empty_like(r)
                for k, qk in enumerate(q):
                    torch.mul(r, float(qk), out=x)
                    x.sin_()
                    x.mul_(ww)
                    out[a, b, k] += x.sum() / float(qk) + extra
            if b > a:
                out[b, a] = out[a, b]
    return out.cpu().numpy()


def _points(case, v, multipole):
    """Points, weights and classes with their three amplitudes: of the atoms, and of the sites where there are any."""
    xyz, element, occupancy, group = v["atoms"]
    names, cls = _classes(element, group)
    q, kind = v["q"], case.get("hydration", "analytic")
    amp = np.array([_amplitudes(e, g, q, multipole) for e, g in names])  # [class, term, q]
    w = occupancy
    if kind in ("none", "adaptive"):
        amp[:, 2] = 0.0
    if kind == "none":
        amp[:, 1] = 0.0
    if kind == "adaptive":
        sites = _shell_sites(xyz, float(case["spacing"]))
        h = np.zeros((1, 3, len(q)))
        h[0, 2] = _water(q, float(case["spacing"]))
        amp = np.concatenate([amp, h])
        xyz, w = np.concatenate([xyz, sites]), np.concatenate([w, np.ones(len(sites))])
        cls = np.concatenate([cls, np.full(len(sites), len(names))])
    return xyz, w, cls, amp


def _scale(q, c1):
    return c1 ** 3 * np.exp(-(c1 * c1 - 1.0) * 1.62 ** 2 * q * q / 4.0)


def _combined(amp, q, kind):
    if kind == "none":
        return amp[:, 0]
    return amp[:, 0] - _scale(q, 1.01) * amp[:, 1] + 1.1 * amp[:, 2]


def _exact_multipole(case, v):
    """The expansion in 64 bits: orders up to l_max, cut at each q by ceil(q R) + 8, R the farthest point."""
    xyz, w, cls, amp = _points(case, v, True)
    q, kind, n = v["q"], case["hydration"], case["atoms"]
    centre = xyz[:n].mean(axis=0)
    d = xyz - centre
    radius = np.sqrt((d * d).sum(axis=1))
    lmax = case.get("l_max") or int(min(64, max(8, math.ceil(q.max() * radius[:n].max()) + 8)))
    dev = _device()
    p = torch.tensor(d, dtype=torch.float64, device=dev)
    r = torch.tensor(radius, dtype=torch.float64, device=dev)
    f = torch.tensor(_combined(amp, q, kind), dtype=torch.float64, device=dev)  # [class, q]
    wt, ct = torch.tensor(w, dtype=torch.float64, device=dev), torch.tensor(cls, device=dev)
    x = p[:, 2] / r.clamp_min(1e-12)
    s = (1.0 - x * x).clamp_min(0.0).sqrt()
    rho = (p[:, 0] ** 2 + p[:, 1] ** 2).sqrt()
    turn = torch.complex(torch.where(rho > 0, p[:, 0] / rho.clamp_min(1e-300), torch.ones_like(rho)),
                         torch.where(rho > 0, p[:, 1] / rho.clamp_min(1e-300), torch.zeros_like(rho)))
    # normalised Legendre functions P[l][m], m >= 0, and the real harmonics from them
    legendre = {(0, 0): torch.full_like(x, math.sqrt(1.0 / (4.0 * math.pi)))}
    for m in range(1, lmax + 1):
        legendre[(m, m)] = -math.sqrt((2 * m + 1) / (2.0 * m)) * s * legendre[(m - 1, m - 1)]
    for m in range(lmax):
        legendre[(m + 1, m)] = math.sqrt(2 * m + 3.0) * x * legendre[(m, m)]
        for l in range(m + 2, lmax + 1):
            a = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
            b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0))
            legendre[(l, m)] = a * (x * legendre[(l - 1, m)] - b * legendre[(l - 2, m)])
    powers = [torch.ones_like(turn)]
    for m in range(lmax):
        powers.append(powers[-1] * turn)
    harmonics = []
    for l in range(lmax + 1):
        cols = [legendre.pop((l, 0))]
        for m in range(1, l + 1):
            y = math.sqrt(2.0) * legendre.pop((l, m))
            cols += [y * powers[m].real, y * powers[m].imag]
        harmonics.append(torch.stack(cols, dim=1))
    out = np.zeros(len(q))
    step = max(1, 40_000_000 // (len(radius) * (lmax + 30)))
    rmax = radius.max()
    lq = np.clip(np.ceil(q * rmax).astype(int) + 8, min(8, lmax), lmax)
    for k0 in range(0, len(q), step):
        qk = torch.tensor(q[k0:k0 + step], dtype=torch.float64, device=dev)
        z = (qk[:, None] * r[None, :]).clamp_min(1e-8)
        fw = f[:, k0:k0 + step].T[:, ct] * wt
        top = int(max(lmax + 24, lq[k0:k0 + step].max() + 24))
        j = [None] * (lmax + 1)
        after, now = torch.zeros_like(z), torch.full_like(z, 1e-250)
        for l in range(top, 0, -1):  # downward recurrence, kept in range
            before = (2.0 * l + 1.0) / z * now - after
            after, now = now, before
            if l - 1 <= lmax:
                j[l - 1] = now
            big = now.abs() > 1e150
            if bool(big.any()):
                k = torch.where(big, torch.full_like(z, 1e-150), torch.ones_like(z))
                now, after = now * k, after * k
                for i in range(min(l - 1, lmax), lmax + 1):
                    if l - 1 <= lmax and j[i] is not None:
                        j[i] = j[i] * k
        j0, j1 = z.sin() / z, z.sin() / (z * z) - z.cos() / z
        k = torch.where(j0.abs() >= j1.abs(), j0 / j[0], j1 / j[1])
        total = torch.zeros(len(qk), dtype=torch.float64, device=dev)
        for l in range(lmax + 1):
            a = (fw * (j[l] * k)) @ harmonics[l]
            on = torch.tensor((lq[k0:k0 + step] >= l).astype(np.float64), device=dev)
            total += on * (a * a).sum(dim=1)
        out[k0:k0 + step] = 4.0 * math.pi * total.cpu().numpy()
    return {"intensity": np.maximum(out, 0.0)}


def _basis(S, amp):
    v, e, h = amp[:, 0], amp[:, 1], amp[:, 2]
    return np.stack([np.einsum("ak,bk,abk->k", x, y, S)
                     for x, y in ((v, v), (e, e), (h, h), (v, e), (v, h), (e, h))])


def _exact_gradient(case, v):
    xyz, w, cls, amp = _points(case, v, False)
    q, y, sigma = v["q"], v["y"], v["sigma"]
    S = _pair_sums(xyz, w, cls, len(amp), q)
    f = _combined(amp, q, "analytic")
    b = _basis(S, amp)
    G, c1, c2 = _scale(q, 1.01), 1.01, 1.1
    intensity = b[0] + G * G * b[1] + c2 * c2 * b[2] - 2 * G * b[3] + 2 * c2 * b[4] - 2 * G * c2 * b[5]
    scale, dof = v["scale"], max(len(q) - 1, 1)
    res = (scale * intensity - y) / sigma
    dm = 2.0 * res / sigma / dof
    dg = G * (3.0 / c1 - 2.0 * c1 * 1.62 ** 2 * q * q / 4.0)
    params = [float((dm * scale * (2 * G * b[1] - 2 * b[3] - 2 * c2 * b[5]) * dg).sum()),
              float((dm * scale * (2 * c2 * b[2] + 2 * b[4] - 2 * G * b[5])).sum()), float((dm * intensity).sum()),
              float(dm.sum())]
    dev = _device()
    p = torch.tensor(xyz, dtype=torch.float64, device=dev)
    a = torch.tensor(f, dtype=torch.float64, device=dev)[torch.tensor(cls, device=dev)] * torch.tensor(
        w, dtype=torch.float64, device=dev)[:, None]  # [atom, q]
    grad = torch.zeros_like(p)
    rows = max(1, 6_000_000 // len(xyz))
    for i in range(0, len(xyz), rows):
        d = p[i:i + rows, None, :] - p[None, :, :]
        r = (d * d).sum(dim=2).sqrt()
        near = r < 1e-9
        rs = r.clamp_min(1e-9)
        h = torch.zeros_like(r)
        for k, qk in enumerate(q):
            x = rs * float(qk)
            h += (2.0 * float(dm[k] * scale)) * (a[i:i + rows, k, None] * a[None, :, k]) * (x.cos() - x.sin() / x)
        h = torch.where(near, torch.zeros_like(h), h / (rs * rs))
        grad[i:i + rows] = (h[:, :, None] * d).sum(dim=1)
    return {"chi2": float((res * res).sum() / dof), "grad_xyz": grad.cpu().numpy(), "grad_params": np.array(params)}


def _exact_pr(case, v):
    xyz, element, occupancy, group = v["atoms"]
    names, cls = _classes(element, group)
    zero = np.zeros(1)
    f0 = np.array([_gauss(_GROUP[g] if g >= 0 else _ELEMENT[e], zero)[0] for e, g in names])
    w = np.maximum(np.abs(occupancy * f0[cls]), 1e-6)
    centre = (xyz * w[:, None]).sum(axis=0) / w.sum()
    rg = math.sqrt((w * ((xyz - centre) ** 2).sum(axis=1)).sum() / w.sum())
    dev = _device()
    p, wt = torch.tensor(xyz, dtype=torch.float64, device=dev), torch.tensor(w, dtype=torch.float64, device=dev)
    rows = max(1, 6_000_000 // len(xyz))

    def squared(i):
        d = p[i:i + rows, None, :] - p[None, :, :]
        return d[..., 0] ** 2 + d[..., 1] ** 2 + d[..., 2] ** 2

    dmax = math.sqrt(max(float(squared(i).max()) for i in range(0, len(xyz), rows)))
    step = dmax / case["bins"]
    hist = torch.zeros(case["bins"], dtype=torch.float64, device=dev)
    for i in range(0, len(xyz), rows):
        k = (squared(i).sqrt() / step).floor().long().clamp_max(case["bins"] - 1)
        at = torch.arange(i, min(i + rows, len(xyz)), device=dev)
        ww = wt[i:i + rows, None] * wt[None, :]
        ww[at - i, at] = 0.0
        hist += torch.bincount(k.reshape(-1), weights=ww.reshape(-1), minlength=case["bins"])
    r = (np.arange(case["bins"]) + 0.5) * step
    h = hist.cpu().numpy() / 2.0
    area = (0.5 * step * (h[1:] + h[:-1])).sum()
    return {"rg": rg, "dmax": dmax, "r": r, "p": h / area}


def exact(case, seed):
    """Debye terms, curves, gradients, P(r) and the adaptive sites in 64 bits.  A fit and an ensemble's weights come
    from iterations, which have no such value; P(r) of over 30,000 atoms takes too long."""
    kind = case["kind"]
    if kind in ("fit", "ensemble"):
        return None
    v = _inputs(case, seed)
    if kind == "grids":
        return {"adaptive": _shell_sites(v["atoms"][0], case["spacing"]), "exterior": None, "volumes": [None, None]}
    if kind == "pr":
        return _exact_pr(case, v) if case["atoms"] <= 30000 else None
    if kind == "gradient":
        return _exact_gradient(case, v)
    if kind == "curve" and case["atoms"] >= 500 or kind == "curve" and case["hydration"] == "adaptive":
        return _exact_multipole(case, v)
    xyz, w, cls, amp = _points(case, v, False)
    S = _pair_sums(xyz, w, cls, len(amp), v["q"])
    if kind == "curve":
        f = _combined(amp, v["q"], case["hydration"])
        return {"intensity": np.maximum(np.einsum("ak,bk,abk->k", f, f, S), 0.0)}
    return {"basis": _basis(S, amp)}
