"""The FP64 atmospheric bins in fixed point: on the CPU (the same source built for the host)
against the oracle over Earth models and parameter sets, with the range test that hands a bin
to the FP64 path; on the GPU at the edges of its launch and of its table kernel."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from cudaprob3_gb300 import earth
from oracle.oracle import Mixing as OMix

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "cudaprob3_gb300", "csrc")
dp = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    so = str(tmp_path_factory.mktemp("fixed") / "libfixed.so")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-shared",
                        "-Xcompiler", "-fPIC,-ffp-contract=off", "-I", SRC,
                        "-I", os.path.join(os.path.dirname(HERE), "include"),
                        os.path.join(HERE, "cpp", "fixed_bins.cu"), os.path.join(SRC, "cp3_host.cpp"), "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return C.CDLL(so)


def host_bins(lib, m, anti, cz, en, model, h, refine=1):
    a = [np.ascontiguousarray(x, dtype=np.float64)
         for x in ([m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq], cz, en, *model)]
    p = [x.ctypes.data_as(dp) for x in a]
    out = np.empty((9, len(cz), len(en)))
    n = lib.fixed_atmos(p[0], -1 if anti else 1, int(anti), p[1], len(cz), p[2], len(en), p[3], p[4], p[5],
                        len(a[3]), C.c_double(h), refine, out.ctypes.data_as(dp))
    return np.transpose(out, (1, 2, 0)), n


def test_float_pairs_and_reciprocals(host):
    """The start of the eigen-solver: a double as a float pair to 2^-48 (a low word of 29 bits
    rounded to 24, below 2^-23), from 2^-60 to 2^61 and nothing else; its reciprocal to a unit and
    a half of the last place; a fixed-point number from a pair to the rounding of 2^-30 2^-24."""
    host.fixed_pair.argtypes = [C.c_double, C.c_void_p, C.c_void_p]
    host.fixed_from_pair.argtypes = [C.c_float, C.c_float]
    host.fixed_from_pair.restype = C.c_longlong
    pair, rec = np.zeros(2, dtype=np.float32), C.c_double()

    def split(x):
        return host.fixed_pair(x, pair.ctypes.data, C.byref(rec))

    rng = np.random.default_rng(13)
    values = np.concatenate([np.exp(rng.uniform(np.log(1e-3), np.log(1e6), 4000)), 2.0 ** np.arange(-60, 61),
                             np.nextafter(2.0 ** np.arange(-59, 62), 0), np.nextafter(2.0 ** np.arange(-60, 61), 1e99)])
    for x in np.concatenate([values, -values]):
        assert split(x), x
        hi, lo = float(pair[0]), float(pair[1])
        assert abs(lo) <= 2.0 ** -24 * abs(hi) * (1 + 2.0 ** -20)
        assert abs((hi - x) + lo) <= 2.0 ** -48 * abs(x)
        assert abs(rec.value * np.longdouble(x) - 1) <= 1.5 * 2.0 ** -52
    for x in (0.0, -0.0):
        assert split(x) and not pair.any()
    for x in (np.nan, np.inf, -np.inf, 2.0 ** 61, 2.0 ** -60 * (1 - 2.0 ** -53), 5e-324, -1e300):
        assert not split(x), x
    for x in np.concatenate([rng.uniform(-1, 1, 4000), [1.0, -1.0, 0.0, 2.0 ** -31, 1e-12]]):
        hi = np.float32(x)
        lo = np.float32(x - float(hi))
        exact = (int(float(hi) * 2.0 ** 80) + int(float(lo) * 2.0 ** 80)) / 2.0 ** 18
        assert abs(host.fixed_from_pair(hi, lo) - exact) <= 2.0 ** (62 - 54) + 1


def omix(m, anti):
    return OMix(m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq, -1 if anti else 1)


def test_trig_table(host):
    t = np.zeros((512, 2), dtype=np.int64)
    host.fixed_trig(t.ctypes.data_as(C.c_void_p))
    a = 2 * np.longdouble("3.14159265358979323846264") * np.arange(512) / 512
    # 2^-53 of the double functions compared with
    assert np.abs(t[:, 0] * 2.0 ** -62 - np.cos(a)).max() <= 4e-16
    assert np.abs(t[:, 1] * 2.0 ** -62 - np.sin(a)).max() <= 4e-16


def test_negation_at_the_low_words_ends(host):
    """-v to one unit for every low word, its lowest value (which has no 32-bit negative) among
    them; a bin in 4e6 met it, 2e-11 off."""
    host.fixed_negated.restype = C.c_longlong
    for high in (0, 1, -1, 12345, -(1 << 30), (1 << 30) - 1):
        for low in (-(1 << 31), -(1 << 31) + 1, -1, 0, 1, (1 << 31) - 1):
            v = high * (1 << 32) + low
            assert abs(host.fixed_negated(C.c_longlong(v)) + v) <= 1


@pytest.mark.parametrize("shells,h", [(1, 22.0), (2, 0.0), (3, 15.0), (12, 22.0), (59, 100.0), (128, 22.0)])
def test_host_bins_against_oracle(host, oracle, shells, h):
    """Both orderings, nu and nubar, vacuum-only rows, vertical and shell-grazing rows, at the
    FP64 parity bar; every bin inside the fixed-point range.  With the eigen-systems from the
    FP64 formulas, and refined in fixed point from vectors cut at 2^-46."""
    model = earth.synthetic_shells(shells)
    cz = np.concatenate([np.linspace(-1, 1, 23), [-1e-9, -0.5]])
    en = np.logspace(-1, 3, 17)
    for m in earth.gaussian_sets(4, seed=7)[1:3]:
        for anti in (False, True):
            ref = oracle.atmos(omix(m, anti), anti, cz, en, *model, h, layer_limit=128)
            for refine in (0, 1):
                got, outside = host_bins(host, m, anti, cz, en, model, h, refine)
                assert outside == 0
                assert np.abs(got - ref).max() <= 1e-12


@pytest.mark.parametrize("shells", [1, 4, 12, 59])
def test_host_bins_against_forty_digits(host, shells):
    """The parity bar of 1e-12 would not see two digits lost.  Against 40-digit arithmetic on the
    same segments a probability is off by twice its phase's error: the rates are rounded four times
    on the way (2.5 2^-52 of the phase, 2.534 |dm| L / E), a layer's sine and cosine are good to
    2^-56, twice a layer and twice through the chain, and the mixing matrix is one of doubles."""
    mp = pytest.importorskip("mpmath").mp.clone()
    mp.dps = 40
    model = earth.synthetic_shells(shells)
    m = earth.gaussian_sets(3, seed=7)[2]
    arrays = [np.ascontiguousarray(x, dtype=np.float64) for x in model]
    cz, en = np.array([-1.0, -0.83, -0.41, -0.05, 0.3]), np.array([0.7, 3.0, 20.0, 150.0])
    O = (mp.matrix([[mp.cos(m.theta13), 0, mp.sin(m.theta13)], [0, 1, 0], [-mp.sin(m.theta13), 0, mp.cos(m.theta13)]]) *
         mp.matrix([[mp.cos(m.theta12), mp.sin(m.theta12), 0], [-mp.sin(m.theta12), mp.cos(m.theta12), 0], [0, 0, 1]]))
    H0 = O * mp.diag([0, mp.mpf(m.dm12sq), mp.mpf(m.dm12sq) + mp.mpf(m.dm23sq)]) * O.T
    for anti in (False, True):
        got, outside = host_bins(host, m, anti, cz, en, model, 22.0)
        assert outside == 0
        W = (mp.matrix([[1, 0, 0], [0, mp.cos(m.theta23), mp.sin(m.theta23)], [0, -mp.sin(m.theta23), mp.cos(m.theta23)]]) *
             mp.diag([1, 1, mp.expj(-m.dcp if anti else m.dcp)]))
        for ie, E in enumerate(en):
            eigen = {}
            for ic, c in enumerate(cz):
                length, rho_e = np.empty(200), np.empty(200)
                n = host.fixed_segments(C.c_double(c), *(x.ctypes.data_as(dp) for x in arrays), len(arrays[0]),
                                        C.c_double(22.0), length.ctypes.data_as(dp), rho_e.ctypes.data_as(dp))

                def layer(l):
                    if l not in eigen:
                        H = H0.copy()
                        H[0, 0] += (-1 if anti else 1) * mp.mpf(1.52588e-4) * mp.mpf(float(E)) * mp.mpf(float(rho_e[l]))
                        eigen[l] = mp.eigsy(H)
                    lam, U = eigen[l]
                    f = mp.mpf(2.534) * mp.mpf(float(length[l])) / mp.mpf(float(E))
                    return U * mp.diag([mp.expj(-(x - lam[0]) * f) for x in lam]) * U.T

                G = mp.eye(3)
                for l in range(1, n - 1):
                    G = layer(l) * G
                G = G.T * layer(n - 1) * G if n > 1 else G
                A = W * G * layer(0) * W.H
                ref = [float(abs(A[b, a]) ** 2) for a in range(3) for b in range(3)]
                total = length[0] + 2 * length[1:n].sum()
                phase = 2.534 * (abs(m.dm12sq) + abs(m.dm23sq) + 1.53e-4 * E * rho_e[:n].max()) * total / E
                assert np.abs(got[ic, ie] - ref).max() <= 2 * (2.5 * 2.0 ** -52 * phase + 4 * n * 2.0 ** -56 + 2e-16), (c, E)


@pytest.mark.parametrize("dm23sq", [1e-10, 2e-11, -1e-11])
def test_nearly_equal_levels_stay_in_fixed_point(host, oracle, dm23sq):
    """Two vacuum levels a millionth of the spread apart: the FP64 vectors of the two are not
    orthogonal after one step, which sent every bin to the FP64 path.  The roots of a nearly double
    level are off by sqrt(2^-53) of the spread, 8e-13 eV^2: 3e-7 rad over 13 000 km at 0.1 GeV."""
    m = earth.NOMINAL
    m = type(m)(m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, dm23sq)
    cz, en = np.linspace(-1, 0.4, 15), np.logspace(-1, 2, 13)
    for anti in (False, True):
        got, outside = host_bins(host, m, anti, cz, en, earth.PREM_4LAYER, 22.0, refine=0)
        assert outside == 0
        assert np.abs(got - oracle.atmos(omix(m, anti), anti, cz, en, *earth.PREM_4LAYER, 22.0)).max() <= 3e-7


@pytest.mark.parametrize("shells", [1, 4, 59, 128])
@pytest.mark.parametrize("theta12,theta13", [(0.0, 0.0), (0.0, 0.15), (0.59, 0.0)])
def test_host_bins_are_probabilities(host, shells, theta12, theta13):
    """Nothing below 0 or above 1 where a channel is exactly zero or one (a decoupled flavour) and
    the rounding of a deep chain could leave it on either side."""
    m = earth.NOMINAL
    m = type(m)(theta12, theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq)
    cz, en = np.linspace(-1, 0.3, 53), np.logspace(-1, 3, 101)
    for anti in (False, True):
        got, outside = host_bins(host, m, anti, cz, en, earth.synthetic_shells(shells), 22.0)
        assert outside == 0
        assert got.min() >= 0.0 and got.max() <= 1.0


def test_out_of_range_bins_ask_for_the_fp64_path(host):
    """Energies that are not finite or zero, and phases past 2^42 turns (13 000 km at 1e-13 GeV
    and below); the neighbouring energies stay inside."""
    cz = np.array([-0.9, 0.5])
    en = np.array([1.0, np.nan, 0.0, np.inf, 1e-16, 5.0])
    with np.errstate(all="ignore"):
        for i in range(len(en)):
            _, outside = host_bins(host, earth.NOMINAL, False, cz, en[i:i + 1], earth.PREM_4LAYER, 22.0)
            assert outside == (0 if i in (0, 5) else len(cz)), en[i]


@pytest.mark.parametrize("poly", [False, True])
@pytest.mark.parametrize("nb,h", [(0, 22.0), (1, 0.0), (3, 22.0), (20, 15.0)])
def test_host_bins_solved_in_place_against_oracle(host, oracle, poly, nb, h):
    """Quadratic densities and production-height averaging: one bin and twenty, wide bins whose
    sinc leaves its series, an air segment of zero length (h = 0); weights that are not a
    distribution ask for the FP64 path."""
    r, abc, ye = ((earth.PREM_4LAYER_QUAD_V2[0], earth.PREM_4LAYER_QUAD_V2[1:4], earth.PREM_4LAYER_QUAD_V2[4]) if poly
                  else (earth.PREM_12LAYER[0], (earth.PREM_12LAYER[1],) * 3, earth.PREM_12LAYER[2]))
    cz, en = np.concatenate([np.linspace(-1, 1, 13), [-0.02]]), np.logspace(-1, 2, 11)
    rng = np.random.default_rng(4)
    edges = np.linspace(2.0, 80.0, nb + 1)
    prob = rng.uniform(0.1, 1.0, (2, 3, len(en), len(cz), max(nb, 1)))
    prob /= prob.sum(axis=-1, keepdims=True)
    m = earth.gaussian_sets(2, seed=9)[1]
    for anti in (False, True):
        ref = oracle.atmos(omix(m, anti), anti, cz, en, r, None if poly else abc[0], ye, h, poly_abc=abc if poly else None,
                           avg=(nb, prob.ravel(), edges) if nb else None)
        for scale, want in ((1.0, 0), (2.0, len(cz) * len(en) if nb else 0)):
            a = [np.ascontiguousarray(x, dtype=np.float64)
                 for x in ([m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq], cz, en, r, *abc, ye,
                           np.transpose(scale * prob, (0, 1, 3, 4, 2)), edges)]
            p = [x.ctypes.data_as(dp) for x in a]
            out = np.empty((9, len(cz), len(en)))
            n = host.fixed_inline(p[0], -1 if anti else 1, int(anti), p[1], len(cz), p[2], len(en), p[3], p[4], p[5], p[6],
                                  p[7], len(r), int(poly), C.c_double(h), nb, p[8], p[9], out.ctypes.data_as(dp))
            assert n == want
            if scale == 1.0:
                assert np.abs(np.transpose(out, (1, 2, 0)) - ref).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("shells,nc,ne", [(1, 1, 1), (1, 5, 33), (7, 4, 32), (8, 3, 31), (9, 6, 64), (16, 9, 65), (128, 13, 40)])
def test_gpu_bins_at_the_edges_of_the_launch(oracle, shells, nc, ne):
    """Rows and energies around a block's four warps of 32, class counts around the table
    kernel's runs of eight, up to the largest model."""
    from tests.gpu_helpers import run_atmos
    model = earth.synthetic_shells(shells)
    cz, en = np.linspace(-1, 0.4, nc), earth.log_energy_grid(ne)
    m = earth.gaussian_sets(2, seed=8)[1]
    mix6 = [m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    for anti in (False, True):
        got = run_atmos("fp64", mix6, -1 if anti else 1, anti, cz, en, *model, 22.0)
        assert np.abs(got - oracle.atmos(omix(m, anti), anti, cz, en, *model, 22.0, layer_limit=128)).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("nb,nc,ne", [(1, 1, 1), (2, 5, 33), (20, 3, 31)])
def test_gpu_averaged_bins_at_the_edges_and_out_of_range(oracle, nb, nc, ne):
    """Averaged bins (FP64 and mixed) at the block edges, with weights that do not add up to one:
    sums up to 1.2 stay in fixed point, sums of 3 take the FP64 path."""
    from tests.test_gpu_averaging import run_avg
    r, rho, ye = earth.synthetic_shells(9)
    cz, en = np.linspace(-1, 0.4, nc), earth.log_energy_grid(ne)
    prob = np.random.default_rng(6).uniform(0.1, 1.0, (2, 3, ne, nc, nb))
    prob /= prob.sum(axis=-1, keepdims=True)
    edges = np.linspace(3.0, 60.0, nb + 1)
    m = earth.gaussian_sets(2, seed=10)[1]
    mix6 = [m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    for scale in (1.0, 1.2, 3.0):
        w = (scale * prob).ravel()
        ref = oracle.atmos(omix(m, True), True, cz, en, r, rho, ye, 20.0, avg=(nb, w, edges))
        for prec, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            got = run_avg(prec, mix6, -1, True, cz, en, r, rho, ye, 20.0, nb, w, edges)
            assert np.abs(got - ref).max() <= tol * max(1.0, scale)


WEIGHT_SUMS = (1.0, 1.25, 1.2500001, 2.5, 3.0, 17.0, 1e6, 0.0, 1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("poly", [False, True])
@pytest.mark.parametrize("nb", [1, 2, 20])
def test_gpu_averaged_bins_with_weights_that_are_no_distribution(oracle, poly, nb):
    """Every cell's weights of a sum of its own, some negative, one cell with a weight that is not
    a number: each cell within the bar times its own sum, the NaN in its own cell alone."""
    from tests.test_gpu_averaging import run_avg
    r, abc, ye = ((earth.PREM_4LAYER_QUAD_V2[0], earth.PREM_4LAYER_QUAD_V2[1:4], earth.PREM_4LAYER_QUAD_V2[4]) if poly
                  else (earth.PREM_12LAYER[0], (earth.PREM_12LAYER[1],) * 3, earth.PREM_12LAYER[2]))
    cz, en = np.linspace(-1, 0.4, 9), earth.log_energy_grid(37)
    rng = np.random.default_rng(11)
    prob = rng.uniform(0.1, 1.0, (2, 3, len(en), len(cz), nb))
    prob /= prob.sum(axis=-1, keepdims=True)
    sums = rng.choice(WEIGHT_SUMS, prob.shape[:-1])
    prob *= sums[..., None]
    prob[:, :, ::3, :, 0] *= -1.0
    edges = np.linspace(3.0, 60.0, nb + 1)
    m = earth.gaussian_sets(2, seed=10)[1]
    mix6 = [m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    args = (r, None if poly else abc[0], ye, 20.0)
    for anti in (False, True):
        ref = oracle.atmos(omix(m, anti), anti, cz, en, *args, poly_abc=abc if poly else None, avg=(nb, prob.ravel(), edges))
        # [cosine][energy][channel], the initial flavour of a channel its cell's
        bar = 1e-12 * np.maximum(1.0, np.repeat(np.transpose(sums[int(anti)], (2, 1, 0)), 3, axis=2))
        run = lambda w: run_avg("fp64", mix6, -1 if anti else 1, anti, cz, en, *args, nb, w.ravel(), edges,
                                abc if poly else None)
        got = run(prob)
        assert (np.abs(got - ref) <= bar).all()
        bad = prob.copy()
        bad[int(anti), 1, 5, 3, 0] = np.nan
        got = run(bad)
        assert np.isnan(got[3, 5, 3:6]).all()
        got[3, 5, 3:6] = ref[3, 5, 3:6]
        assert (np.abs(got - ref) <= bar).all()


@pytest.mark.gpu
def test_gpu_weights_that_are_no_distribution_run_on_the_common_kernel():
    """They cost what a distribution's cost (the FP64 path took ten times that)."""
    import time
    from cudaprob3_gb300 import AtmosCudaPropagatorSingle
    nc, ne, nb, m = 200, 150, 20, earth.NOMINAL
    best = {}
    for scale in (1.0, 3.0):
        p = AtmosCudaPropagatorSingle(0, nc, ne, precision="fp64")
        p.setEnergyList(earth.log_energy_grid(ne))
        p.setCosineList(earth.cosine_grid(nc))
        p.setMNSMatrix(m.theta12, m.theta13, m.theta23, m.dcp, 1)
        p.setNeutrinoMasses(m.dm12sq, m.dm23sq)
        p.setDensity(*earth.PREM_12LAYER)
        p.setProductionHeight(22.0)
        p.SetNumberOfProductionHeightBinsForAveraging(nb)
        p.setProductionHeightList(np.full(6 * nc * ne * nb, scale / nb), np.linspace(5.0, 45.0, nb + 1))
        times = []
        for _ in range(20):
            t = time.perf_counter()
            p.calculateProbabilities(0)
            times.append(time.perf_counter() - t)
        best[scale] = min(times)
    assert best[3.0] < 3.0 * best[1.0], best


@pytest.mark.gpu
@pytest.mark.parametrize("shells", [59, 128])
@pytest.mark.parametrize("nb", [0, 1, 20])
def test_gpu_results_are_probabilities(shells, nb):
    """As test_host_bins_are_probabilities, plain bins and bins averaged with weights that add up
    to one."""
    from tests.gpu_helpers import run_atmos
    from tests.test_gpu_averaging import run_avg
    m = earth.NOMINAL
    mix6 = [0.0, 0.0, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    cz, en = np.linspace(-1, 0.3, 53), np.logspace(-1, 3, 101)
    w = np.random.default_rng(3).uniform(0.1, 1.0, (2, 3, len(en), len(cz), max(nb, 1)))
    w /= w.sum(axis=-1, keepdims=True)
    model = earth.synthetic_shells(shells)
    for anti in (False, True):
        if nb:
            got = run_avg("fp64", mix6, -1 if anti else 1, anti, cz, en, *model, 22.0, nb, w.ravel(),
                          np.linspace(5.0, 45.0, nb + 1))
        else:
            got = run_atmos("fp64", mix6, -1 if anti else 1, anti, cz, en, *model, 22.0)
        assert got.min() >= 0.0 and got.max() <= 1.0


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 2, 20])
def test_gpu_averages_with_negative_weights(oracle, nb):
    """Weights below zero can take an averaged value out of [0, 1], which it keeps."""
    from tests.test_gpu_averaging import run_avg
    cz, en = np.linspace(-1, 0.4, 7), earth.log_energy_grid(33)
    prob = np.random.default_rng(12).uniform(0.1, 1.0, (2, 3, len(en), len(cz), nb))
    prob /= prob.sum(axis=-1, keepdims=True)
    prob[:, :, ::2, :, 0] *= -1.0
    edges = np.linspace(3.0, 60.0, nb + 1)
    m = earth.gaussian_sets(2, seed=10)[1]
    mix6 = [m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    ref = oracle.atmos(omix(m, False), False, cz, en, *earth.PREM_4LAYER, 20.0, avg=(nb, prob.ravel(), edges))
    assert ref.min() < -0.01 or nb == 20  # (with twenty it stays inside)
    got = run_avg("fp64", mix6, 1, False, cz, en, *earth.PREM_4LAYER, 20.0, nb, prob.ravel(), edges)
    assert np.abs(got - ref).max() <= 1e-12


@pytest.mark.gpu
def test_gpu_out_of_range_bins():
    """A NaN energy gives NaN in its own column and leaves the others as they are.  An energy too
    low for the fixed-point reduction takes the FP64 path: its phases (1e18 rad) have lost every
    digit there, so the values only have to be finite."""
    from tests.gpu_helpers import run_atmos
    m = earth.NOMINAL
    mix6 = [m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq]
    cz, en = np.linspace(-1, 0.4, 7), earth.log_energy_grid(40)
    ok = run_atmos("fp64", mix6, 1, False, cz, en, *earth.PREM_4LAYER, 22.0)
    en[5], en[37] = np.nan, 1e-16
    got = run_atmos("fp64", mix6, 1, False, cz, en, *earth.PREM_4LAYER, 22.0)
    keep = [i for i in range(40) if i not in (5, 37)]
    assert np.array_equal(got[:, keep], ok[:, keep])
    assert np.isnan(got[:, 5]).all()
    assert np.isfinite(got[:, 37]).all()
