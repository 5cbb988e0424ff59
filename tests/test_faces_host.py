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
#include <cstring>
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
static inline int __float_as_int(float x) { int i; memcpy(&i, &x, 4); return i; }
static inline float __int_as_float(int i) { float x; memcpy(&x, &i, 4); return x; }
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

// the fast speeds of single states (dimension 1), as the HLL / HLLC sweeps and as the HLLD sweeps take them
extern "C" void speeds32(int n, const float *P, float *out)
{
  for (int i = 0; i < n; ++i, P += 8, out += 4) {
    float U[8], F[8];
    prim_to_cons(4.f / 3.f, P, U);
    flux_and_eigenvalues(4.f / 3.f, U, P, F, out[0], out[1], 1);
    SideState s, t;
    float ml = 0.f;
    face_sides(4.f / 3.f, P, P, P[Bx], s, t, out[2], out[3], ml);
  }
}

// the first rung of the zone c2p, as the FP64 path (accurate) and as the FP32-bulk path (fast) runs it
extern "C" void c2p(int n, const double *U, double *accurate, double *fast, int *err)
{
  for (int i = 0; i < n; ++i, U += 8, accurate += 8, fast += 8) {
    C2PState s;
    s.gamma = 4.0 / 3.0;
    s.gamf = 0.25;
    s.pfloor = -1.0;
    c2p_new_state(s, U);
    double Z, W;
    int it;
    c2p_estimate(s, Z, W);
    err[2 * i] = c2p_anton2dzw(s, Z, W, accurate, it);
    err[2 * i + 1] = c2p_anton2dzw_fast(s, Z, W, fast, it);
  }
}

// minmod of slope triples: 32 the FP32 form, 64 the reference's expression
extern "C" void minmod(int n, const float *abc, float *f32, double *f64)
{
  for (int i = 0; i < n; ++i, abc += 3) {
    f32[i] = minmod3(abc[0], abc[1], abc[2]);
    f64[i] = minmod3(double(abc[0]), double(abc[1]), double(abc[2]));
  }
}

// a face's outer speeds (dimension 1)
extern "C" void face_speeds32(int n, const float *pl, const float *pr, float *out)
{
  for (int i = 0; i < n; ++i, pl += 8, pr += 8, out += 2) {
    SideState s, t;
    float ml = 0.f;
    face_sides(4.f / 3.f, pl, pr, pl[Bx], s, t, out[0], out[1], ml);
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
    L.speeds32.argtypes = [ctypes.c_int, _f, _f]
    L.c2p.argtypes = [ctypes.c_int, _d, _d, _d, _i]
    L.minmod.argtypes = [ctypes.c_int, _f, _f, _d]
    L.face_speeds32.argtypes = [ctypes.c_int, _f, _f, _f]
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


@pytest.mark.parametrize("scale", [1e-10, 1e-9, 1e-8, 1e-7, 1e-6, 1e-4, 1e-2, 1e2, 1e4, 1e5, 1e6, 1e7, 1e8])
def test_pressures_far_from_one_fall_back_to_hllc_where_the_oracle_does(lib, scale):
    """The reference's difference step is an absolute 1e-8: at pressures far above one its slopes
    are rounding, far below one they are not local, and its own iteration alone tells which
    faces it rejects."""
    P, Q = random_faces(5000, 2.0, 0.3)
    for X in (P, Q):
        X[:, :2] *= scale
        X[:, 5:] *= np.sqrt(scale)
    F0, e0, u0 = oracle_hlld(P, Q)
    F, e, u = host_hlld(lib, P, Q)
    assert np.array_equal(e, e0) and np.array_equal(u, u0)
    assert face_rel(F, F0)[e0 == 0].max() <= 1e-10


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


# ---- FP32 fast speeds ---------------------------------------------------------------------------

def fast_speeds(P):
    """The extreme roots (largest, smallest) of the fast magnetosonic quartic of the states P
    (direction 1), in extended precision:
      rho h (1 - cs^2) W^4 d^4 = (1 - l^2) ((b^2 + rho h cs^2) W^2 d^2 - cs^2 (b^x - l b^0)^2),
    l = v + d, in units of d / s with s^2 = cs^2 + b^2 / rho h.  From outside the roots, Newton's
    iteration falls onto them monotonically."""
    P = P.astype(np.longdouble)
    rho, p, v, vB = P[:, 0], P[:, 1], P[:, 2], (P[:, 2:5] * P[:, 5:]).sum(1)
    iW2 = 1 - (P[:, 2:5] ** 2).sum(1)
    rh = rho + p * 4
    cs2, b2 = GAMMA * p / rh, (P[:, 5:] ** 2).sum(1) * iW2 + vB ** 2
    s2 = cs2 + b2 / rh
    s = np.sqrt(s2)
    w = P[:, 5] * iW2                       # (b^x - l b^0) / W = w - d vB
    out = []
    for sg in (1, -1):
        def f(x):
            d = s * x
            return (1 - cs2) / iW2 * x ** 4 - (1 - (v + d) ** 2) * (x ** 2 - cs2 / rh * ((w - d * vB) / s2) ** 2)
        x = sg * (1 + np.abs(v)) / s        # outside |l| = 1
        x = sg * np.minimum(np.abs(x), 1 / s + 2)
        for _ in range(60):
            h = np.abs(x) * np.longdouble(1e-9)
            df = (f(x + h) - f(x - h)) / (2 * h)
            x = x - f(x) / df
        out.append((v + s * x).astype(np.float64))
    return out


def cold_states():
    rng = np.random.default_rng(3)
    rows = []
    for p in 10.0 ** np.arange(-36, 1, 2):
        for v in ((0.0, 0.0, 0.0), (0.1, 0.2, 0.1), (-0.6, 0.3, 0.2)):
            for B in ((0.3, 0.1, 0.2), (1e-3, 1e-3, 2e-3), (0.0, 0.5, 0.0), (2.0, -1.0, 0.5)):
                rows.append((1.0, p) + v + tuple(b * rng.uniform(0.8, 1.2) for b in B))
    return np.array(rows, dtype=np.float32)


def test_fp32_speeds_down_to_the_coldest_gas(lib):
    """Coefficients rounded to some 1e-7 and roots that are simple: 1e-5 allows for a condition of
    a hundred."""
    P = cold_states()
    out = np.zeros((len(P), 4), np.float32)
    lib.speeds32(len(P), P, out)
    hi, lo = fast_speeds(P)
    for k in (0, 2):
        assert np.abs(out[:, k] - hi).max() <= 1e-5, (k, P[np.abs(out[:, k] - hi).argmax()])
        assert np.abs(out[:, k + 1] - lo).max() <= 1e-5, (k, P[np.abs(out[:, k + 1] - lo).argmax()])


@pytest.mark.parametrize("angle,jump,dv", [(0.01, 0.1, 0.02), (0.05, 0.02, 0.02), (0.02, 0.05, 0.01)])
def test_fp32_outer_speeds_where_fast_and_slow_meet(lib, angle, jump, dv):
    """Faces with the field nearly along the sweep and Alfven and sound speeds nearly equal: the
    fast and slow roots of a side almost coincide, and each side's iteration must end at its
    own fast root, wherever it is started from.  Rounding of 1e-7 in the coefficients moves a double
    root by the square root of that: 1e-3 allows for a condition of ten."""
    rng = np.random.default_rng(11)
    n = 4000
    p, rho = np.exp(rng.uniform(np.log(0.1), np.log(10), n)), np.exp(0.1 * rng.standard_normal(n))
    rh = rho + 4 * p
    cs2 = GAMMA * p / rh
    B = np.sqrt(rh * cs2 / (1 - cs2) * np.exp(0.1 * rng.standard_normal(n)))   # Alfven speed ~ sound speed
    th, ph = angle * rng.random(n), 2 * np.pi * rng.random(n)
    P = np.stack([rho, p] + [0.01 * rng.standard_normal(n) for _ in range(3)] +
                 [B * np.cos(th), B * np.sin(th) * np.cos(ph), B * np.sin(th) * np.sin(ph)], axis=1)
    Q = P * (1 + jump * rng.standard_normal((n, 8)) * np.array([1, 1, 0, 0, 0, 0, 1, 1]))
    Q[:, 2:5] += dv * rng.standard_normal((n, 3))
    P, Q = P.astype(np.float32), Q.astype(np.float32)
    out = np.zeros((n, 2), np.float32)
    lib.face_speeds32(n, P, Q, out)
    l, r = fast_speeds(P), fast_speeds(Q)
    assert np.abs(out[:, 0] - np.maximum(l[0], r[0])).max() <= 1e-3
    assert np.abs(out[:, 1] - np.minimum(l[1], r[1])).max() <= 1e-3


def test_fp32_minmod_is_the_reference_expression(lib):
    """PLM slopes of three zones, any of which may be NaN."""
    rng = np.random.default_rng(5)
    v = rng.choice(np.array([-2.0, -1.0, -0.5, 0.0, 0.25, 1.0, 3.0, np.nan], np.float32), (20000, 3))
    abc = np.stack([2 * (v[:, 1] - v[:, 0]), 0.5 * (v[:, 2] - v[:, 0]), 2 * (v[:, 2] - v[:, 1])], axis=1)
    f32, f64 = np.zeros(len(v), np.float32), np.zeros(len(v))
    lib.minmod(len(v), np.ascontiguousarray(abc, dtype=np.float32), f32, f64)
    assert np.isnan(f64).any() and np.array_equal(f32, f64.astype(np.float32), equal_nan=True)


# ---- the FP32-bulk c2p --------------------------------------------------------------------------

@pytest.mark.parametrize("wmax,plo,phi", [(1.5, 0.1, 10.0), (3.0, 0.1, 10.0), (3.0, 1e-3, 1e-2)])
def test_fp32_bulk_c2p_ends_at_fp64_accuracy(lib, wmax, plo, phi):
    """Both iterations end on a step below 1e-12, with an error of that step's square and the
    rounding of the conserved state, some 1e-15 of Z = rho h W^2, which p inherits: ten times
    that.  Where the first rung fails it fails for both."""
    rng = np.random.default_rng(4)
    P, _ = random_faces(4000, wmax, 0.0)
    P[:, 1] = P[:, 0] * np.exp(rng.uniform(np.log(plo), np.log(phi), len(P)))
    port = PortOracle(Scheme(n=(4, 4, 4)))
    U = np.array([port.prim_to_cons(p)[0] for p in P])
    A, B, e = np.zeros_like(U), np.zeros_like(U), np.zeros(2 * len(U), np.int32)
    lib.c2p(len(U), U, A, B, e)
    ok = e[::2] == 0
    assert np.array_equal(e[::2], e[1::2]) and ok.mean() > 0.97
    Z = (P[:, 0] + 4 * P[:, 1]) / (1 - (P[:, 2:5] ** 2).sum(1))
    assert (np.abs(A[:, 1] - B[:, 1]) / Z)[ok].max() <= 1e-14
