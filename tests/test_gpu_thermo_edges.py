"""The fixed-scratch statmech reduction at the edges of its split (warps, blocks, chunks) and of its
exponential's range, against the same sums in extended precision on the host."""
import ctypes as C

import numpy as np
import pytest

from flexaidds_gb300 import capi, evaluator

pytestmark = pytest.mark.gpu

BLOCKS, THREADS, CHUNK = 4 * 152, 256, 8


def _energies(n, kind):
    rng = np.random.default_rng(n)
    if kind == "descending":        # every chunk brings a new largest weight
        return np.sort(rng.normal(-30.0, 6.0, n))[::-1].copy()
    e = rng.normal(-30.0, 6.0, n)
    if kind == "wide":              # weights from 1 to below the smallest double, and two infinities
        e = rng.uniform(-40.0, 1500.0, n)
        e[:: max(1, n // 2)] = -40.0
        if n > 4:
            e[3] = e[n - 2] = np.inf
    return e


@pytest.mark.parametrize("kind", ["plain", "descending", "wide"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, BLOCKS * THREADS - 1, BLOCKS * THREADS + 1,
                               BLOCKS * THREADS * CHUNK, BLOCKS * THREADS * CHUNK + 33])
def test_fixed_scratch_reduction_against_extended_precision(n, kind):
    torch = pytest.importorskip("torch")
    lib = evaluator.load_library()
    lib.fxe_thermo_compute_device_fixed.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_double, C.c_void_p, C.c_void_p]
    e = _energies(n, kind)
    T = 310.0
    de, out = torch.from_numpy(e).cuda(), torch.zeros(C.sizeof(capi.Thermo), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.fxe_thermo_compute_device_fixed(de.data_ptr(), None, n, T, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    t = capi.Thermo.from_buffer_copy(out.cpu().numpy().tobytes())
    x = e[np.isfinite(e)].astype(np.longdouble)
    beta = np.longdouble(1.0 / (0.001987206 * T))
    lw = -beta * x
    w = np.exp(lw - lw.max())
    s = w.sum()
    log_z, mean, sq = float(lw.max() + np.log(s)), float((w * x).sum() / s), float((w * x * x).sum() / s)
    # |lw| <= 130 where weights count: a log-weight rounds by 1.5e-14, a weight so by as much relatively;
    # sums of at most 60 roundings in a chain add 7e-15
    tol = 1e-13
    assert abs(t.log_Z - log_z) <= tol * max(1.0, abs(log_z))
    assert abs(t.mean_energy - mean) <= tol * max(1.0, abs(mean))
    assert abs(t.mean_energy_sq - sq) <= tol * max(1.0, sq)
    kT = 0.001987206 * T
    assert abs(t.heat_capacity - (sq - mean * mean) / kT ** 2) <= 4 * tol * max(1.0, sq) / kT ** 2


@pytest.mark.parametrize("kind", ["plain", "descending", "wide"])
@pytest.mark.parametrize("n", [1, 33, 255, 257, BLOCKS * THREADS - 1, BLOCKS * THREADS + 1, BLOCKS * THREADS * CHUNK + 33])
def test_fixed_scratch_reduction_with_multiplicities(n, kind):
    """The form with multiplicities at the same edges; from 1 to the largest, and infinite energies."""
    torch = pytest.importorskip("torch")
    lib = evaluator.load_library()
    lib.fxe_thermo_compute_device_fixed.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_double, C.c_void_p, C.c_void_p]
    e = _energies(n, kind)
    rng = np.random.default_rng(n + 1)
    mult = rng.integers(1, 100, n).astype(np.int32)
    mult[rng.integers(0, n, max(1, n // 50))] = np.iinfo(np.int32).max
    T = 310.0
    de, dm = torch.from_numpy(e).cuda(), torch.from_numpy(mult).cuda()
    out = torch.zeros(C.sizeof(capi.Thermo), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.fxe_thermo_compute_device_fixed(de.data_ptr(), dm.data_ptr(), n, T, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    t = capi.Thermo.from_buffer_copy(out.cpu().numpy().tobytes())
    fin = np.isfinite(e)
    x = e[fin].astype(np.longdouble)
    beta = np.longdouble(1.0 / (0.001987206 * T))
    lw = np.log(mult[fin].astype(np.longdouble)) - beta * x
    w = np.exp(lw - lw.max())
    s = w.sum()
    log_z, mean, sq = float(lw.max() + np.log(s)), float((w * x).sum() / s), float((w * x * x).sum() / s)
    # as above: the logarithm of a multiplicity, below 22, adds a rounding of 4e-15 to a log-weight
    tol = 1e-13
    assert abs(t.log_Z - log_z) <= tol * max(1.0, abs(log_z))
    assert abs(t.mean_energy - mean) <= tol * max(1.0, abs(mean))
    assert abs(t.mean_energy_sq - sq) <= tol * max(1.0, sq)
    kT = 0.001987206 * T
    assert abs(t.heat_capacity - (sq - mean * mean) / kT ** 2) <= 4 * tol * max(1.0, sq) / kT ** 2


@pytest.mark.parametrize("where", [0, 700, 2047, 2500])
@pytest.mark.parametrize("with_mult", [False, True])
@pytest.mark.parametrize("value", [np.nan, -np.nan, -np.inf])
def test_not_a_number_and_minus_infinity_reach_the_record(value, with_mult, where):
    """A NaN or an infinitely low energy makes the whole record NaN, wherever it stands."""
    torch = pytest.importorskip("torch")
    lib = evaluator.load_library()
    lib.fxe_thermo_compute_device_fixed.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_double, C.c_void_p, C.c_void_p]
    e = np.random.default_rng(1).normal(-30.0, 5.0, 2501)
    e[where] = value
    de = torch.from_numpy(e).cuda()
    dm = torch.full((len(e),), 3, dtype=torch.int32, device="cuda") if with_mult else None
    out = torch.zeros(8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.fxe_thermo_compute_device_fixed(de.data_ptr(), dm.data_ptr() if with_mult else None, len(e), 300.0,
                                               out.data_ptr(), None) == 0
    assert np.isnan(out.cpu().numpy()[1:4]).all()
