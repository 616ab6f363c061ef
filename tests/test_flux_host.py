"""The FP32-bulk interior face fluxes on the host (tests/flux_host_check.cpp compiles dndsg_bodies.cuh as
plain C++): the flux-difference Roe and HLLC forms, FP64 means and central flux with FP32 increments,
jumps and wave terms (face_flux_roe_delta32, face_flux_hllc_delta32), against the FP64 face_flux on the
same face data (the same coefficients and basis record, 3 Gauss points, positivity fallback), over
20,000 random faces per case.

The point of the flux-difference form: every FP32 rounding scales with the reconstruction increment or
the jump across the face, not with the flux.  On a smooth field (jumps and increments of 1e-3) the FP32
flux therefore agrees with FP64 below FP32's own resolution of the flux (measured 1.4e-8 to 2.4e-8 of
the flux).  Across strong jumps (density and pressure ratios up to 25, velocity jumps of the order of
the sound speed, Mach up to 2) the agreement is that of FP32 on the jump (measured at most 7e-6 for Roe
and 1.5e-5 for HLLC, median 5e-8).  Faces whose Gauss points either path sends to the positivity
fallback are left out of the bound (the fallback is a threshold decision; a few dozen faces of the
strong-jump case).  Outside this regime (Mach 5 at near-vacuum pressure, or wave-speed estimates that do
not bracket the contact) FP32 storage itself loses digits, by about Mach^2 in the pressure."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GAMMA = 1.4


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("flux") / "flux_host_check.so"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "dnds_b200", "csrc"),
                        os.path.join(ROOT, "tests", "flux_host_check.cpp"), "-o", str(so)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(str(so))
    L.flux_check.restype = C.c_int
    L.flux_check.argtypes = [C.c_int64, C.c_int] + [C.c_void_p] * 6 + [C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


def _cells(rng, n, jump, mach):
    """Left states with density 0.3-2, pressure 0.2-2 and Mach up to `mach`; right states with density and
    pressure ratios up to 5^jump either way and a velocity jump of `jump` sound speeds (Mach capped)."""
    rho, p = rng.uniform(0.3, 2.0, n), rng.uniform(0.2, 2.0, n)
    a = np.sqrt(GAMMA * p / rho)
    th, M = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, mach, n)
    u, v = M * a * np.cos(th), M * a * np.sin(th)
    ratio = lambda: np.exp(jump * rng.uniform(-1, 1, n) * np.log(5.0))
    rho2, p2 = rho * ratio(), p * ratio()
    a2 = np.sqrt(GAMMA * p2 / rho2)
    u2, v2 = u + jump * a * rng.normal(0, 1, n), v + jump * a * rng.normal(0, 1, n)
    cap = np.maximum(np.sqrt(u2 ** 2 + v2 ** 2) / (mach * a2), 1.0)
    u2, v2 = u2 / cap, v2 / cap

    def cons(r, u, v, p):
        return np.stack([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)], 1)

    U = np.empty((2 * n, 4))
    U[0::2], U[1::2] = cons(rho, u, v, p), cons(rho2, u2, v2, p2)
    return np.ascontiguousarray(U)


def _run(lib, riemann, jump, inc, seed, n=20000):
    rng = np.random.default_rng(seed)
    U = _cells(rng, n, jump, 2.0)
    urec = np.ascontiguousarray(rng.normal(0, inc, (2 * n, 20)).astype(np.float32))
    basis = np.ascontiguousarray(rng.uniform(-1, 1, (n, 18)).astype(np.float32))
    th = rng.uniform(0, 2 * np.pi, n)
    N = np.ascontiguousarray(np.stack([np.cos(th), np.sin(th)], 1))
    area, dlam = np.ascontiguousarray(rng.uniform(0.5, 2, n)), np.ascontiguousarray(rng.uniform(0, 0.5, n))
    err, scale, red = np.zeros(n), np.zeros(n), np.zeros(n, np.int32)
    flagged = lib.flux_check(n, riemann, U.ctypes.data, urec.ctypes.data, basis.ctypes.data, N.ctypes.data,
                             area.ctypes.data, dlam.ctypes.data, GAMMA, err.ctypes.data, scale.ctypes.data,
                             red.ctypes.data)
    assert flagged == 0
    kept = red == 0
    return err[kept] / scale[kept], int((~kept).sum())


@pytest.mark.parametrize("riemann", [1, 2], ids=["roe", "hllc"])
def test_smooth_field_below_fp32_resolution(lib, riemann):
    rel, reduced = _run(lib, riemann, 1e-3, 1e-3, seed=10 + riemann)
    assert reduced == 0
    assert rel.max() < 6e-8, rel.max()


@pytest.mark.parametrize("riemann", [1, 2], ids=["roe", "hllc"])
def test_strong_jumps_within_fp32_of_the_jump(lib, riemann):
    rel, reduced = _run(lib, riemann, 1.0, 0.02, seed=20 + riemann)
    assert reduced < 200
    assert rel.max() < 5e-5, rel.max()
    assert np.median(rel) < 2e-7, np.median(rel)


def test_positivity_fallback_as_the_quotient_form(lib):
    """CompressRecPart (DNDS_FV_EulerEvaluator.hpp:1277-1360) without its quotient: the mean where density or
    E - |m|^2 / (2 (rho + 1e-200)) is negative, and the state as it is, not finite, where an entry is NaN (the flux then
    flags it).  Zero and infinite entries too, one per state."""
    rng = np.random.default_rng(3)
    n = 40000
    um = np.stack([rng.uniform(0.1, 2, n), rng.normal(0, 1, n), rng.normal(0, 1, n), rng.uniform(1, 5, n)], 1)
    inc = um * rng.normal(0, 0.7, (n, 4))
    at = np.arange(0, n, 4)
    inc[at, rng.integers(0, 4, at.size)] = rng.choice([np.nan, np.inf, -np.inf], at.size)
    zero = np.arange(1, n, 16)
    k = rng.integers(0, 4, zero.size)
    inc[zero, k] = -um[zero, k]
    r, red = np.empty((n, 4)), np.empty(n, np.int32)
    lib.compress_check.argtypes = [C.c_int64] + [C.c_void_p] * 4
    lib.compress_check.restype = None
    lib.compress_check(n, um.ctypes.data, inc.ctypes.data, r.ctypes.data, red.ctypes.data)
    with np.errstate(all="ignore"):
        want = um + inc
        low = want[:, 0] < 0
        want[low] = um[low]
        kin = 0.5 * (want[:, 1] ** 2 + want[:, 2] ** 2) / (want[:, 0] + 1e-200)
        cold = want[:, 3] - kin < 0
        want[cold] = um[cold]
        tie = np.abs(want[:, 3] - kin) < 1e-12 * np.abs(kin)  # a rounding decides
    assert not tie.any() and low.sum() > 1000 and cold.sum() > 1000
    assert np.array_equal(red != 0, low | cold)
    assert np.array_equal(r, want, equal_nan=True)
