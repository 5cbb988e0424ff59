"""The per-face and per-zone device functions of the sweeps and the c2p, compiled for the host
(g++, no FMA contraction) and held to the C restatement or to plain FP64 arithmetic, on states
that turbulence boxes do not reach: high Lorentz factors, weak normal fields, cold gas.

Flux bounds are relative to the face's largest flux component."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import PortOracle, Scheme

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "ctf_b200", "csrc")
GAMMA = 4.0 / 3.0

PROGRAM = r"""
#include <cmath>
#include <cuda_runtime.h>
#undef __noinline__
#define __noinline__ __attribute__((noinline))
#undef __forceinline__
#define __forceinline__ inline
using std::isnan; using std::isinf; using std::isfinite;
static inline float rsqrtf(float x) { return 1.f / sqrtf(x); }
static inline float __fdividef(float a, float b)   // CUDA's delivers 0 above 2^126
{
  return fabsf(b) > 8.507059e37f ? 0.f * a : a / b;
}
#include "rmhd_face32.cuh"
namespace mgpu { bool c2p_learned_guess(const void *, const C2PState &, double &, double &) { return false; } }
using namespace mgpu;

static PhysParams params()
{
  PhysParams pp{};
  pp.gamma = 4.0 / 3.0;
  pp.pfloor = -1.0;
  return pp;
}

extern "C" void hlld64(int n, const int *dim, const double *pl, const double *pr, double *F, int *err, int *hllc)
{
  for (int i = 0; i < n; ++i, pl += 8, pr += 8, F += 8) {
    double states[32], f[8] = {0}, ml = 0.0;
    for (int q = 0; q < 8; ++q) {
      states[q] = pl[frame_slot(dim[i], q)];
      states[8 + q] = pr[frame_slot(dim[i], q)];
    }
    const auto src = [&](double *l, double *r) {
      for (int q = 0; q < 8; ++q) { l[q] = pl[q]; r[q] = pr[q]; }
    };
    C2PTally t{0, 0};
    err[i] = riemann_hlld64(params(), dim[i], Column<double>{states, 1}, f, ml, hllc[i], &t, src);
    for (int q = 0; q < 8; ++q) F[frame_slot(dim[i], q)] = f[q];
  }
}
"""

_i, _d, _f = (np.ctypeslib.ndpointer(dtype=t, flags="C_CONTIGUOUS") for t in (np.int32, np.float64, np.float32))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = next((p for p in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda",
                             os.path.join(os.path.dirname(shutil.which("nvcc") or ""), ".."))
                 if os.path.exists(os.path.join(p, "include", "cuda_runtime.h"))), None)
    if cuda is None or shutil.which("g++") is None:
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("faces")
    (d / "faces.cpp").write_text(PROGRAM)
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I", CSRC, "-I",
                        os.path.join(cuda, "include"), str(d / "faces.cpp"), "-o", str(d / "faces.so")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    L = ctypes.CDLL(str(d / "faces.so"))
    L.hlld64.argtypes = [ctypes.c_int, _i, _d, _d, _d, _i, _i]
    return L


# ---- states ----------------------------------------------------------------------------------

def random_faces(n, wmax, jump, bn=None, seed=7):
    """Faces of direction 1 with Lorentz factors up to wmax, order-one density, pressure and
    field, every component but the normal field differing by a random `jump`; bn: the normal
    field's magnitude (None: of order one)."""
    rng = np.random.default_rng(seed)
    W = 1 + (wmax - 1) * rng.random(n)
    d = rng.standard_normal((n, 3))
    P = np.empty((n, 8))
    P[:, :2] = np.exp(0.5 * rng.standard_normal((n, 2)))
    P[:, 2:5] = d / np.linalg.norm(d, axis=1, keepdims=True) * np.sqrt(1 - 1 / W ** 2)[:, None]
    P[:, 5:] = rng.standard_normal((n, 3))
    if bn is not None:
        P[:, 5] = bn * (1 + rng.random(n))
    k = jump * rng.standard_normal((n, 8))
    k[:, 5] = 0
    Q = P * (1 + k)
    Q[:, :2] = np.abs(Q[:, :2])
    sp, mx = np.linalg.norm(Q[:, 2:5], axis=1, keepdims=True), 1 - 0.5 / wmax ** 2
    Q[:, 2:5] *= np.where(sp > mx, mx / sp, 1.0)
    return P, Q


# K_R and K_L meet on the way of this face's pressure iteration
MEETING = (np.array([[1.17211, 2.66462, -0.0165776, 0.548085, 0.834274, 6.85834, -0.997862, -2.44169]]),
           np.array([[0.532589, 3.52797, 0.0111665, 0.856906, 0.512891, 6.85834, -1.13433, -3.28915]]))


def oracle_hlld(P, Q, **kw):
    """Flux, error and whether the face fell back to HLLC, of the C restatement."""
    port = PortOracle(Scheme(n=(4, 4, 4), riemann="hlld"), **kw)
    F, e, u = np.zeros_like(P), np.zeros(len(P), dtype=int), np.zeros(len(P), dtype=bool)
    for i in range(len(P)):
        F[i], e[i] = port.riemann(P[i], Q[i], 1)
        u[i] = port.stats.hlld_path in (0, 4)
    return F, e, u


def host_hlld(lib, P, Q):
    n = len(P)
    F, e, u = np.zeros((n, 8)), np.zeros(n, np.int32), np.zeros(n, np.int32)
    lib.hlld64(n, np.ones(n, np.int32), P, Q, F, e, u)
    return F, e, u != 0


def face_rel(A, B):
    return np.abs(A - B).max(axis=1) / np.abs(B).max(axis=1)


# ---- FP64 HLLD ---------------------------------------------------------------------------------

@pytest.mark.parametrize("wmax", [10.0, 50.0])
def test_relativistic_jumps_fall_back_to_hllc_where_the_oracle_does(lib, wmax):
    """Where K_R and K_L meet, equation 48's residual is zero by definition; the reference
    rejects such an attempt, and most of these faces end in HLLC."""
    P, Q = random_faces(3000, wmax, 0.5)
    P, Q = np.concatenate([MEETING[0], P]), np.concatenate([MEETING[1], Q])
    F0, e0, u0 = oracle_hlld(P, Q)
    F, e, u = host_hlld(lib, P, Q)
    assert u0[0] and u0.sum() > 100
    assert np.array_equal(e != 0, e0 != 0)
    assert np.array_equal(u, u0), np.flatnonzero(u != u0)
    ok = e0 == 0
    assert face_rel(F[ok], F0[ok]).max() <= 1e-10   # the whole-step bound, face by face


@pytest.mark.parametrize("wmax", [1.5, 3.0, 10.0])
@pytest.mark.parametrize("bn", [2e-8, 1e-7, 1e-6])
def test_weak_normal_fields_keep_the_oracle_bits(lib, wmax, bn):
    """Equation 48's residual scales with the normal field, so that at |Bx| far below sqrt(p) it
    passes wherever the iteration starts: only the reference's own start and iteration give
    its flux, and they give every bit of it."""
    P, Q = random_faces(2000, wmax, 0.05, bn)
    F0, e0, u0 = oracle_hlld(P, Q)
    F, e, u = host_hlld(lib, P, Q)
    assert np.array_equal(e, e0) and np.array_equal(u, u0)
    assert np.array_equal(F[e0 == 0], F0[e0 == 0])


@pytest.mark.parametrize("bn", [1e-3, 3e-3])
def test_small_normal_fields_are_iterated_to_the_oracle_accuracy(lib, bn):
    """The pressure ends within the slope's last few percent of a step of 4e-12 (2e-13), and the
    residual's rounding (1e-16 of the Alfven speeds, whose difference is of the order of the
    normal field) adds 1e-16 / bn (1e-13): 5e-13 allows for both and the fluxes' own rounding."""
    P, Q = random_faces(40000, 20.0, 0.02, bn)
    F0, e0, u0 = oracle_hlld(P, Q)
    F, e, u = host_hlld(lib, P, Q)
    assert np.array_equal(e, e0) and np.array_equal(u, u0)
    ok = e0 == 0
    assert face_rel(F[ok], F0[ok]).max() <= 5e-13
