"""The workloads this library is timed on: what its users have it compute, through its public
entry points, over the sizes its configurations, tests and benchmark use.

A case is a dict of plain values.  ``prepare`` builds what a user's program holds before a
call (propagators, batches or a server with their grids and Earth model set), ``run`` is one
evaluation at one oscillation-parameter set per problem, as a fit step makes it, ``work`` its
necessary traffic and arithmetic, and ``exact`` the same probabilities from plain numpy and
torch in 64 bits.
"""
import math

import numpy as np
import torch

from cudaprob3_gb300 import AtmosCudaPropagatorSingle, BeamCudaPropagatorSingle, earth
from cudaprob3_gb300.batch import Batch
from cudaprob3_gb300.serve import Server
from cudaprob3_gb300.types import Mixing

HEIGHT_KM = earth.PRODUCTION_HEIGHT_KM
BEAM_RHO = 2.6


def listed():
    return [
        # The drop-in call on the default grid and model: 400 x 400 bins, PREM with four
        # shells, FP64.  A small call, where launches and latency count.
        dict(name="atmos_fp64_prem4", kind="atmos", precision="fp64", model="prem4", nc=400, ne=400, anti=0),
        # The drop-in call on an uneven, odd-sized grid and the finer PREM, antineutrinos.
        dict(name="atmos_fp64_prem12_ragged", kind="atmos", precision="fp64", model="prem12", nc=307, ne=811, anti=1),
        # The largest single grid, FP64: 59 shells, 2000 x 2000 bins.
        dict(name="atmos_fp64_shells59", kind="atmos", precision="fp64", model="shells59", nc=2000, ne=2000, anti=0),
        # The same grid in mixed precision, neutrinos and antineutrinos, queued as a fitter
        # with two propagators queues them.
        dict(name="atmos_mixed_shells59", kind="atmos_pair", precision="mixed", model="shells59", nc=2000, ne=2000),
        # A small mixed evaluation whose result the caller reads on the host.
        dict(name="atmos_mixed_to_host", kind="to_host", precision="mixed", model="prem4", nc=200, ne=200, anti=0),
        # Quadratic density inside the shells (a density of its own in every segment).
        dict(name="atmos_fp64_quadratic", kind="atmos", precision="fp64", model="quadratic", nc=500, ne=500, anti=0),
        # Production-height averaging over 20 height bins.
        dict(name="atmos_fp64_averaged", kind="averaged", precision="fp64", model="prem4", nc=200, ne=150, bins=20, anti=0),
        # A long baseline, FP64: 1e5 energies.
        dict(name="beam_fp64", kind="beam", precision="fp64", ne=100000, length_km=1300.0, anti=0),
        # A short energy list in mixed precision: the smallest call.
        dict(name="beam_mixed_small", kind="beam", precision="mixed", ne=10000, length_km=295.0, anti=1),
        # A fit's parameter sets on uneven grids in one batch (cosines uniform on [100, 1000],
        # energies on [100, 2000], PREM with twelve shells).
        dict(name="batch_atmos", kind="batch_atmos", problems=32, model="prem12", cos_hi=1000, e_hi=2000),
        # Beam parameter sets at two baselines in one batch.
        dict(name="batch_beam", kind="batch_beam", problems=64, baselines=2, ne=100000),
        # A burst of requests of mixed sizes to the server, waited for.
        dict(name="serve_burst", kind="serve", requests=32, model="prem4"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["atmos", "atmos", "atmos", "atmos_pair", "to_host", "averaged", "beam", "beam",
                       "batch_atmos", "batch_beam", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    anti = rng.randrange(2)
    model = rng.choice(["prem4", "prem12", "shells59"])
    if kind == "atmos":
        if rng.random() < 0.3:  # every segment solves its own eigen-system: smaller grids
            return dict(kind=kind, precision=precision, model="quadratic", nc=_log_int(rng, 40, 1000),
                        ne=_log_int(rng, 40, 1000), anti=anti)
        return dict(kind=kind, precision=precision, model=model, nc=_log_int(rng, 40, 2000),
                    ne=_log_int(rng, 40, 2000), anti=anti)
    if kind == "atmos_pair":
        return dict(kind=kind, precision="mixed", model=model, nc=_log_int(rng, 100, 2000), ne=_log_int(rng, 100, 2000))
    if kind == "to_host":
        return dict(kind=kind, precision=precision, model=model, nc=_log_int(rng, 50, 1000), ne=_log_int(rng, 50, 1000),
                    anti=anti)
    if kind == "averaged":
        return dict(kind=kind, precision=precision, model=rng.choice(["prem4", "prem12", "quadratic"]),
                    nc=_log_int(rng, 30, 300), ne=_log_int(rng, 30, 300), bins=rng.randint(1, 20), anti=anti)
    if kind == "beam":
        return dict(kind=kind, precision=precision, ne=_log_int(rng, 100, 200000),
                    length_km=round(rng.uniform(200.0, 1500.0), 1), anti=anti)
    if kind == "batch_atmos":
        return dict(kind=kind, problems=rng.randint(2, 40), model=rng.choice(["prem4", "prem12"]),
                    cos_hi=_log_int(rng, 200, 1000), e_hi=_log_int(rng, 200, 2000))
    if kind == "batch_beam":
        return dict(kind=kind, problems=2 * rng.randint(1, 32), baselines=rng.randint(1, 3), ne=_log_int(rng, 1000, 100000))
    return dict(kind="serve", requests=rng.randint(4, 60), model=rng.choice(["prem4", "prem12"]))


# ---- inputs ----------------------------------------------------------------------------

def _model(name):
    """(radii, rho, ye, None) or, with quadratic densities, (radii, None, ye, (a, b, c))."""
    if name == "quadratic":
        r, a, b, c, ye = earth.PREM_4LAYER_QUAD_V2
        return r, None, ye, (a, b, c)
    r, rho, ye = {"prem4": lambda: earth.PREM_4LAYER, "prem12": lambda: earth.PREM_12LAYER,
                  "shells59": lambda: earth.synthetic_shells(59)}[name]()
    return r, rho, ye, None


def _mixing(rng):
    """A parameter set of a fit: Gaussian around the nominal one, either mass ordering."""
    c = earth.NOMINAL
    g = rng.standard_normal(6)
    dm23 = c.dm23sq * (1.0 + 0.03 * g[5])
    return Mixing(float(c.theta12 + 0.02 * g[0]), float(c.theta13 + 0.02 * g[1]), float(c.theta23 + 0.02 * g[2]),
                  float(c.dcp + g[3]), float(c.dm12sq * (1.0 + 0.03 * g[4])),
                  float(-abs(dm23) if rng.random() < 0.5 else dm23))


def _points(rng, n, lo, hi):
    """One point in each of n equal bins of [lo, hi], ascending."""
    return lo + (hi - lo) * (np.arange(n) + rng.uniform(0.2, 0.8, n)) / n


def _cosines(rng, n):
    return _points(rng, n, -1.0, 1.0)


def _energies(rng, n):
    return np.exp(_points(rng, n, math.log(0.1), math.log(100.0)))


def _beam_energies(rng, n):
    return _points(rng, n, 0.1, 10.0)


_BASELINES = (295.0, 1300.0, 810.0)
_SERVE_GRIDS = (("atmos", 200, 200), ("atmos", 500, 500), ("atmos", 2000, 2000), ("beam", 1, 10000), ("beam", 1, 100000))


def _serve_grid_of(rng, n):
    """The grids of a burst: the sizes in equal shares, the largest one at most twice."""
    pick = rng.integers(0, len(_SERVE_GRIDS), n)
    large = np.flatnonzero(pick == 2)
    pick[large[2:]] = 1
    return [int(g) for g in pick]


def _batch_sizes(case):
    """The uneven grids of a batch (its own, the same for every seed)."""
    return earth.uneven_grids(case["problems"], seed=case["problems"] + case["cos_hi"] + case["e_hi"],
                              cos_range=(100, case["cos_hi"]), e_range=(100, case["e_hi"]))


def _inputs(case, seed):
    """Everything random of a case, from the seed alone (prepare and exact share it)."""
    rng = np.random.default_rng(seed)
    k = case["kind"]
    if k in ("atmos", "atmos_pair", "to_host"):
        return dict(cz=_cosines(rng, case["nc"]), en=_energies(rng, case["ne"]), mix=_mixing(rng))
    if k == "averaged":
        nb = case["bins"]
        w = rng.uniform(0.2, 1.0, (2, 3, case["ne"], case["nc"], nb))
        w /= w.sum(axis=-1, keepdims=True)
        return dict(cz=_cosines(rng, case["nc"]), en=_energies(rng, case["ne"]), mix=_mixing(rng), prob=w,
                    edges=np.linspace(5.0, 45.0, nb + 1) + rng.uniform(-0.2, 0.2, nb + 1))
    if k == "beam":
        return dict(en=_beam_energies(rng, case["ne"]), mix=_mixing(rng))
    if k == "batch_atmos":
        return dict(problems=[dict(cz=_cosines(rng, nc), en=_energies(rng, ne), mix=_mixing(rng), anti=p % 2)
                              for p, (nc, ne) in enumerate(_batch_sizes(case))])
    if k == "batch_beam":
        return dict(en=_beam_energies(rng, case["ne"]),
                    problems=[dict(mix=_mixing(rng), anti=p % 2) for p in range(case["problems"])])
    grids = []
    for kind, rows, ne in _SERVE_GRIDS:
        grids.append((_cosines(rng, rows), _energies(rng, ne)) if kind == "atmos" else (None, _beam_energies(rng, ne)))
    which = _serve_grid_of(np.random.default_rng(case["requests"]), case["requests"])  # the same load for every seed
    return dict(grids=grids, requests=[dict(grid=g, mix=_mixing(rng), anti=i % 2) for i, g in enumerate(which)])


# ---- the framework's calls -------------------------------------------------------------

class _DeviceArray:
    """A result in device memory, for torch.as_tensor; it keeps the handle that owns the
    memory for as long as the tensor lives."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=tuple(shape), typestr=typestr, version=3)


def _on_device(owner, ptr, shape, is_float):
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, "<f4" if is_float else "<f8"), device="cuda")


def _atmos(case, x):
    p = AtmosCudaPropagatorSingle(0, case["nc"], case["ne"], precision=case["precision"])
    p.setEnergyList(x["en"])
    p.setCosineList(x["cz"])
    radii, rho, ye, abc = _model(case["model"])
    if abc is None:
        p.setDensity(radii, rho, ye)
    else:
        p.setDensity(radii, *abc, ye)
    p.setProductionHeight(HEIGHT_KM)
    return p


def prepare(case, seed):
    x = _inputs(case, seed)
    k = case["kind"]
    s = dict(kind=k, x=x, anti=case.get("anti", 0))
    if k in ("atmos", "to_host", "averaged"):
        p = s["p"] = _atmos(case, x)
        shape = (9, case["nc"], case["ne"])
        if k == "averaged":
            p.SetNumberOfProductionHeightBinsForAveraging(case["bins"])
            p.setProductionHeightList(x["prob"].ravel(), x["edges"])
        if k == "to_host":
            dt = torch.float32 if case["precision"] == "mixed" else torch.float64
            s["host"] = torch.empty(shape, dtype=dt, pin_memory=True)
        ptr, is_float, _ = p.device_result()
        s["out"] = _on_device(p, ptr, shape, is_float)
    elif k == "atmos_pair":
        s["pair"] = [_atmos(case, x) for _ in range(2)]
        s["out"] = [_on_device(p, p.device_result()[0], (9, case["nc"], case["ne"]), True) for p in s["pair"]]
    elif k == "beam":
        p = s["p"] = BeamCudaPropagatorSingle(0, case["ne"], 1, precision=case["precision"])
        p.setEnergyList(x["en"])
        p.setDensity(BEAM_RHO)
        p.setPathLength(case["length_km"])
        ptr, is_float, _ = p.device_result()
        s["out"] = _on_device(p, ptr, (9, case["ne"]), is_float)
    elif k in ("batch_atmos", "batch_beam"):
        b = s["b"] = Batch(0)
        # a fixed tile shape, which the autotuner finds for batches of this kind: tuning here
        # would take longer than every run it serves
        b.set_shape(16, 0, 16)
        if k == "batch_atmos":
            radii, rho, ye, _ = _model(case["model"])
            b.set_earth(radii, rho, ye, HEIGHT_KM)
            for q in x["problems"]:
                b.set_params(b.add_atmos(q["cz"], q["en"]), q["mix"], bool(q["anti"]))
            shapes = [(9, len(q["cz"]), len(q["en"])) for q in x["problems"]]
        else:
            for q in x["problems"]:
                b.set_params(b.add_beam(x["en"], BEAM_RHO, list(_BASELINES[:case["baselines"]])), q["mix"], bool(q["anti"]))
            shapes = [(case["baselines"], 9, case["ne"])] * case["problems"]
        b.commit()
        s["out"] = [_on_device(b, b.result_ptr(i)[0], shape, True) for i, shape in enumerate(shapes)]
    else:
        v = s["v"] = Server(0, pool_bytes=2 << 30)
        radii, rho, ye, _ = _model(case["model"])
        v.set_earth(radii, rho, ye, HEIGHT_KM)
        for (cz, en) in x["grids"]:
            if cz is not None:
                v.add_atmos_grid(cz, en)
            else:
                v.add_beam_grid(en, BEAM_RHO, [1300.0])
        v.start()
        s["held"] = []
    return s


def _set(p, mix, anti):
    p.setMNSMatrix(mix.theta12, mix.theta13, mix.theta23, mix.dcp, -1 if anti else 1)
    p.setNeutrinoMasses(mix.dm12sq, mix.dm23sq)


def run(s):
    """One evaluation.  The single propagators get their parameter set again, as every fit
    step sets one; a batch's is part of it."""
    k, x = s["kind"], s["x"]
    if k in ("atmos", "averaged", "beam"):
        _set(s["p"], x["mix"], s["anti"])
        s["p"].calculateProbabilities(s["anti"])  # returns when the probabilities are there
        return s["out"]
    if k == "atmos_pair":
        for anti, p in enumerate(s["pair"]):
            _set(p, x["mix"], anti)
            p.calculate_async(anti)
        return s["out"]
    if k == "to_host":
        _set(s["p"], x["mix"], s["anti"])
        s["p"].calculate_to_host_async(s["anti"], s["host"].data_ptr())
        s["p"].synchronize()
        return s["host"]
    if k in ("batch_atmos", "batch_beam"):
        for i, q in enumerate(x["problems"]):
            s["b"].set_params(i, q["mix"], bool(q["anti"]))
        s["b"].run()
        return s["out"]
    v = s["v"]
    for rid in s["held"]:  # the last burst's results are done with
        v.release(rid)
    s["held"] = [v.submit(q["grid"], q["mix"], bool(q["anti"])) for q in x["requests"]]
    out = []
    for rid, q in zip(s["held"], x["requests"]):
        v.wait(rid)
        kind, rows, ne = _SERVE_GRIDS[q["grid"]]
        out.append(_on_device(v, v.result_ptr(rid)[0], (9, rows, ne) if kind == "atmos" else (rows, 9, ne), True))
    return out


# ---- necessary work --------------------------------------------------------------------

def _shells(model, cz):
    radii = np.asarray(_model(model)[0], dtype=np.float64)
    lim = np.sort(-np.sqrt(1.0 - (radii / 6371.0) ** 2))
    lim[-1] = 0.0
    return (np.asarray(cz)[:, None] < lim[None, :]).sum(axis=1)


def _atmos_work(model, nc, ne, size, averaged_bins=0):
    # A bin: two phases with sine and cosine and one 3 x 3 layer for each of its segments
    # (about 100 and 100 operations), and the nine moduli; an eigen-system (about 200) for
    # each class and energy, or for each segment of a bin with quadratic densities.
    seg = _shells(model, (np.arange(nc) + 0.5) / nc * 2 - 1) + 1
    classes = int(seg.max())
    bins = nc * ne
    eigen = float(seg.sum()) * ne if model == "quadratic" else float(classes) * ne
    flops = 200.0 * float(seg.sum()) * ne + 60.0 * bins + 200.0 * eigen + 100.0 * averaged_bins * bins
    return dict(bytes=9.0 * size * bins + 8.0 * (nc + ne) + 3.0 * size * averaged_bins * bins, flops=flops)


def _beam_work(baselines, ne, size):
    return dict(bytes=9.0 * size * baselines * ne + 8.0 * ne, flops=(200.0 + 160.0 * baselines) * ne)


def _add(parts):
    parts = list(parts)
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


def work(case):
    k = case["kind"]
    size = 4 if case.get("precision", "mixed") == "mixed" else 8
    if k in ("atmos", "to_host"):
        return _atmos_work(case["model"], case["nc"], case["ne"], size)
    if k == "averaged":
        return _atmos_work(case["model"], case["nc"], case["ne"], size, case["bins"])
    if k == "atmos_pair":
        return _add([_atmos_work(case["model"], case["nc"], case["ne"], size)] * 2)
    if k == "beam":
        return _beam_work(1, case["ne"], size)
    if k == "batch_atmos":
        return _add(_atmos_work(case["model"], nc, ne, 4) for nc, ne in _batch_sizes(case))
    if k == "batch_beam":
        return _add([_beam_work(case["baselines"], case["ne"], 4)] * case["problems"])
    parts = []
    for g in _serve_grid_of(np.random.default_rng(case["requests"]), case["requests"]):
        kind, rows, ne = _SERVE_GRIDS[g]
        parts.append(_atmos_work(case["model"], rows, ne, 4) if kind == "atmos" else _beam_work(1, ne, 4))
    return _add(parts)


# ---- the same probabilities in 64 bits -------------------------------------------------
# Diagonalised Hamiltonians and ordered 3 x 3 products, in numpy and torch alone.

_GF = 1.52588e-4   # 2 sqrt(2) G_F N_e E per (g / cm^3) GeV, eV^2
_PHASE = 2.534     # 1 / (2 hbar c), GeV / (eV^2 km)
_R = 6371.0


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _vacuum(mix, anti):
    """(O, mu, W): the Hamiltonian times 2E is W (O diag(mu) O^T + V e0 e0^T) W^+."""
    dcp = -mix.dcp if anti else mix.dcp
    s12, c12, s13, c13 = math.sin(mix.theta12), math.cos(mix.theta12), math.sin(mix.theta13), math.cos(mix.theta13)
    s23, c23 = math.sin(mix.theta23), math.cos(mix.theta23)
    O = np.array([[c13, 0, s13], [0, 1, 0], [-s13, 0, c13]]) @ np.array([[c12, s12, 0], [-s12, c12, 0], [0, 0, 1]])
    W = np.array([[1, 0, 0], [0, c23, s23], [0, -s23, c23]]) @ np.diag([1, 1, np.exp(1j * dcp)])
    return O, np.array([0.0, mix.dm12sq, mix.dm12sq + mix.dm23sq]), W


def _eigen(mix, anti, en, rho_e):
    """Eigenvalues relative to the first as phase rates (rad / km) and eigenvectors, for
    electron densities and energies that broadcast together."""
    O, mu, _ = _vacuum(mix, anti)
    en, rho_e = np.broadcast_arrays(en, rho_e)
    H = np.broadcast_to((O * mu) @ O.T, en.shape + (3, 3)).copy()
    H[..., 0, 0] += (-1.0 if anti else 1.0) * _GF * en * rho_e
    lam, vec = np.linalg.eigh(H)
    return _PHASE * (lam - lam[..., :1]) / en[..., None], vec


def _segments(radii, rho, ye, abc, cosz, height_km):
    """Lengths (km) and electron densities of a trajectory's segments: the air, then the
    shells inwards to the innermost one crossed.  Radii outermost first.  The lengths are
    formed as the library documents them (in cm, from differences of squares): at grazing
    incidence their rounding is part of the input."""
    R, h = _R * 1.0e5, height_km * 1.0e5
    path = math.sqrt((R + h) * (R + h) - (R * R) * (1 - cosz * cosz)) - R * cosz
    lim = [0.0] + [-math.sqrt(1 - r * r / (_R * _R)) for r in radii[1:]]
    M = sum(cosz < x for x in lim)
    if cosz >= 0:
        return [path / 1.0e5], [0.0]
    low = _R * _R * (1 - cosz * cosz)
    chord = [2.0 * math.sqrt(max(radii[i] * radii[i] - low, 0.0)) for i in range(M)]
    cm = [path - -2.0 * cosz * R]
    for i in range(M):
        cm.append((0.5 * (chord[i] - chord[i + 1]) if i + 1 < M else chord[i]) * 1.0e5)
    dens = [0.0]
    for i in range(M):
        if abc is None:
            dens.append(rho[i] * ye[i])
            continue
        # the mean of a r^2 + b r + c along the half chord [t0, t1] from the perigee (the
        # innermost segment: the whole chord); r^2 = low + t^2
        a, b, c = (float(v[i]) for v in abc)
        t1 = 0.5 * chord[i]
        t0 = 0.5 * chord[i + 1] if i + 1 < M else 0.0
        if low == 0.0:
            t0 = radii[i + 1] if i + 1 < len(radii) else 0.0

        def integral(t):
            q = math.sqrt(low + t * t)
            lin = 0.5 * (t * q + (low * math.log(t + q) if low > 0.0 else 0.0))
            return a * (low * t + t ** 3 / 3.0) + b * lin + c * t

        dens.append((integral(t1) - integral(t0)) / (t1 - t0) * ye[i])
    return [x / 1.0e5 for x in cm], dens


def _exact_atmos(model, mix, anti, cz, en, averaged=None):
    """[9][nc][ne], channel 3 a + b the probability of a -> b."""
    dev = _device()
    radii, rho, ye, abc = _model(model)
    flip = slice(None, None, -1) if radii[1] > radii[0] else slice(None)
    radii, ye = radii[flip], ye[flip]
    rho = None if rho is None else rho[flip]
    abc = None if abc is None else tuple(v[flip] for v in abc)
    rows = [_segments(radii, rho, ye, abc, float(c), HEIGHT_KM) for c in cz]
    W = torch.tensor(_vacuum(mix, anti)[2], device=dev)
    tables = {}

    def layer(l, members):
        """Eigenvectors [1 or rows][ne][3][3] and phase rates of segment l of some rows."""
        if abc is None:
            if l not in tables:
                om, vec = _eigen(mix, anti, en, rows[members[0]][1][l])
                tables[l] = torch.tensor(vec[None], device=dev), torch.tensor(om[None], device=dev)
            return tables[l]
        om, vec = _eigen(mix, anti, en[None, :], np.array([rows[i][1][l] for i in members])[:, None])
        return torch.tensor(vec, device=dev), torch.tensor(om, device=dev)

    out = torch.empty((9, len(cz), len(en)), dtype=torch.float64, device=dev)
    groups = {}
    for i, r in enumerate(rows):
        groups.setdefault(len(r[0]) - 1, []).append(i)
    for M, every in groups.items():
        step = max(1, 2_000_000 // len(en))
        for at in range(0, len(every), step):
            members = every[at:at + step]
            chain = None  # the layers 1 .. M-1, the last leftmost
            for l in range(M + 1):
                vec, om = layer(l, members)
                L = torch.tensor([rows[i][0][l] for i in members], device=dev, dtype=torch.float64)[:, None, None]
                e = torch.exp(-1j * om * L)
                S = (vec * e[..., None, :]) @ vec.transpose(-1, -2).to(e.dtype)
                if l == 0:
                    air, air_vec, air_om, air_e = S, vec, om, e
                elif l < M:
                    chain = S if chain is None else S @ chain
            if M == 0:
                G = torch.eye(3, dtype=W.dtype, device=dev).expand(len(members), len(en), 3, 3)
            elif M == 1:
                G = S
            else:
                G = chain.transpose(-1, -2) @ (S @ chain)
            if averaged is None:
                A = W @ (G @ air) @ W.conj().T
                P = A.real ** 2 + A.imag ** 2  # [row][ne][final][initial]
            else:
                P = _averaged(G, air_vec, air_om, air_e, W, averaged, anti, members, cz, rows, dev)
            out[:, members, :] = P.permute(3, 2, 0, 1).reshape(9, len(members), len(en))
            del chain, S, G
    return out


def _averaged(G, vec, om, e, W, averaged, anti, members, cz, rows, dev):
    """The probabilities with the air segment's eigencomponents smeared over the production
    heights: each cross term of two eigenstates is weighted by the mean of e^{i d x} over
    path-length shifts x, a sum over height bins of prob sinc(d w / 2) e^{i d m}."""
    prob, edges = averaged
    R = _R * 1.0e5

    def shift(c):
        path = [math.sqrt((R + h) * (R + h) - (R * R) * (1 - c * c)) - R * c for h in [HEIGHT_KM * 1.0e5] + [1.0e5 * x for x in edges]]
        return [(v - path[0]) / 1.0e5 for v in path[1:]]

    sh = torch.tensor([shift(float(cz[i])) for i in members], device=dev, dtype=torch.float64)
    mid, wid = 0.5 * (sh[:, 1:] + sh[:, :-1]), sh[:, 1:] - sh[:, :-1]
    w = torch.tensor(np.ascontiguousarray(prob[1 if anti else 0][:, :, members, :]), device=dev)  # [3][ne][row][bin]
    Wd = W.conj().T
    parts = [W @ ((G @ (vec[..., :, k:k + 1] * e[..., None, k:k + 1])) @ vec[..., :, k:k + 1].transpose(-1, -2).to(e.dtype)) @ Wd
             for k in range(3)]
    P = sum(p.real ** 2 + p.imag ** 2 for p in parts)
    for k in range(3):
        for q in range(k):
            d = -(om[..., k] - om[..., q])  # rad per km, [1 or rows][ne]
            f = torch.zeros((3,) + P.shape[:2], dtype=torch.complex128, device=dev)
            for b in range(mid.shape[1]):
                x = 0.5 * d * wid[:, b:b + 1]
                # the library's sinc, as it documents it: the series for every |x| < 1
                sinc = torch.where(x.abs() < 1.0, 1.0 - x * x / 6.0 + x ** 4 / 120.0, torch.sin(x) / torch.where(x == 0, 1.0, x))
                f += (sinc * torch.exp(1j * d * mid[:, b:b + 1]))[None] * w[..., b].transpose(-1, -2)
            cross = parts[q].conj() * parts[k] * f.permute(1, 2, 0)[:, :, None, :]  # the factor is the initial flavour's
            P = P + 2.0 * cross.real
    return P


def _exact_beam(mix, anti, en, lengths_km):
    """[baselines][9][ne]"""
    dev = _device()
    om, vec = _eigen(mix, anti, en, BEAM_RHO * 0.5)
    om, vec = torch.tensor(om, device=dev), torch.tensor(vec, device=dev).to(torch.complex128)
    W = torch.tensor(_vacuum(mix, anti)[2], device=dev)
    out = []
    for L in lengths_km:
        e = torch.exp(-1j * om * L)
        A = W @ (vec * e[:, None, :]) @ vec.transpose(-1, -2) @ W.conj().T
        out.append((A.real ** 2 + A.imag ** 2).permute(2, 1, 0).reshape(9, len(en)))
    return torch.stack(out)


def exact(case, seed):
    x = _inputs(case, seed)
    k = case["kind"]
    if k in ("atmos", "to_host"):
        return _exact_atmos(case["model"], x["mix"], case["anti"], x["cz"], x["en"])
    if k == "averaged":
        return _exact_atmos(case["model"], x["mix"], case["anti"], x["cz"], x["en"], (x["prob"], x["edges"]))
    if k == "atmos_pair":
        return [_exact_atmos(case["model"], x["mix"], anti, x["cz"], x["en"]) for anti in (0, 1)]
    if k == "beam":
        return _exact_beam(x["mix"], case["anti"], x["en"], [case["length_km"]])[0]
    if k == "batch_atmos":
        return [_exact_atmos(case["model"], q["mix"], q["anti"], q["cz"], q["en"]) for q in x["problems"]]
    if k == "batch_beam":
        return [_exact_beam(q["mix"], q["anti"], x["en"], _BASELINES[:case["baselines"]]) for q in x["problems"]]
    out = []
    for q in x["requests"]:
        cz, en = x["grids"][q["grid"]]
        if cz is None:
            out.append(_exact_beam(q["mix"], q["anti"], en, [1300.0]))
        else:
            out.append(_exact_atmos(case["model"], q["mix"], q["anti"], cz, en))
    return out
