"""The sweeps at the sizes where their tiling can go wrong -- rows shorter and longer than a
block of the z sweep (126 zones per block), the smallest box, columns that do not fill a block
-- and the FP32 reconstruction and wave speeds against the FP64 restatement."""
import numpy as np
import pytest

from ctf_b200 import ics
from ctf_b200.mara import Scheme, Solver
from oracle import PortOracle, Scheme as OScheme
from tests.test_gpu_fp32 import L1_TOL, rel_errors

pytestmark = pytest.mark.gpu


def box(n, seed):
    """Turbulence with density and pressure fluctuations (every component varies)."""
    rng = np.random.default_rng(seed)
    P = ics.turbulence_box(n, seed=seed, vrms=0.3)
    inner = P[3:-3, 3:-3, 3:-3]
    inner[..., :2] = np.exp(0.1 * rng.standard_normal(inner.shape[:3] + (2,)))
    return ics.with_guards(np.ascontiguousarray(inner))


@pytest.mark.parametrize("layout,precision", [("lean", "fp32"), ("lean", "fp64"), ("standard", "fp32"), ("standard", "fp64")])
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 3, 126), (3, 5, 125), (9, 17, 33), (35, 6, 4)])
def test_a_shifted_box_advances_to_the_shifted_result(n, layout, precision):
    """Periodic boxes: where a zone lies in its row, block or chunk must not matter, so the
    advance of the shifted box is the shifted advance, bit for bit."""
    for extrap, riemann, shift in (("plm", "hlld", (1, 2, 1)), ("weno5", "hlld", (2, 1, n[2] // 2)), ("pcm", "hllc", (1, 1, 2))):
        sch = Scheme(precision=precision, layout=layout, extrap=extrap, riemann=riemann, advance="rk2")
        inner = box(n, 5)[3:-3, 3:-3, 3:-3]
        out = []
        for k in ((0, 0, 0), shift):
            s = Solver(sch, n)
            s.upload(ics.with_guards(np.ascontiguousarray(np.roll(inner, k, axis=(0, 1, 2)))))
            assert s.advance(0.1 / max(n)) == 0
            out.append(s.download()[3:-3, 3:-3, 3:-3])
        assert np.array_equal(np.roll(out[0], shift, axis=(0, 1, 2)), out[1]), (extrap, riemann)


def smooth_box(n, seed):
    """Turbulence on a density and pressure that vary by factors of order one over the box: every
    component's reconstruction is resolved, and none is trivial."""
    P = ics.turbulence_box(n, seed=seed, vrms=0.3)
    inner = P[3:-3, 3:-3, 3:-3]
    x, y, z = np.meshgrid(*[(np.arange(m) + 0.5) / m * 2 * np.pi for m in n], indexing="ij")
    inner[..., 0] = np.exp(0.3 * np.sin(x + 2 * y) + 0.2 * np.cos(z))
    inner[..., 1] = np.exp(0.3 * np.cos(2 * x - z) + 0.2 * np.sin(y))
    return ics.with_guards(np.ascontiguousarray(inner))


@pytest.mark.parametrize("IS", ["js96", "b08", "sz10"])
@pytest.mark.parametrize("layout", ["lean", "standard"])
def test_fp32_weno_indicators_match_the_oracle_in_every_component(IS, layout):
    """One step with another indicator differs by 6e-4 or more in every component; FP32 is held to
    a twelfth of that."""
    n, tol = (10, 9, 8), 5e-5
    P0, out = smooth_box(n, 9), {}
    for mode in ("js96", "b08", "sz10"):
        kw = dict(extrap="weno5", IS=mode, riemann="hlld", advance="single")
        cpu, out[mode] = PortOracle(OScheme(n=n, **kw)), P0.copy()
        assert cpu.advance(out[mode], 0.02) == 0
    s = Solver(Scheme(precision="fp32", layout=layout, extrap="weno5", IS=IS, riemann="hlld", advance="single"), n)
    s.upload(P0.copy())
    assert s.advance(0.02) == 0
    P = s.download()
    assert rel_errors(P, out[IS], 3)[0].max() <= tol
    for mode in out:
        assert mode == IS or rel_errors(P, out[mode], 3)[0].min() > 5 * tol, mode


@pytest.mark.parametrize("IS", ["js96", "b08", "sz10"])
@pytest.mark.parametrize("riemann", ["hll", "hllc", "hlld"])
def test_fp32_weno_indicators_match_the_oracle(IS, riemann):
    n = (10, 9, 8)
    kw = dict(extrap="weno5", IS=IS, riemann=riemann, advance="single")
    P0 = ics.turbulence_box(n, seed=9, vrms=0.1)
    cpu, Pc = PortOracle(OScheme(n=n, **kw)), P0.copy()
    assert cpu.advance(Pc, 0.005) == 0
    s = Solver(Scheme(precision="fp32", layout="lean", **kw), n)
    s.upload(P0.copy())
    assert s.advance(0.005) == 0
    l1, _ = rel_errors(s.download(), Pc, 3)
    assert l1[:2].max() <= L1_TOL, l1


def test_fp32_speeds_of_hot_fast_and_field_free_states():
    """MaxLambda of FP32 single steps against FP64 on uniform boxes, where the exact speed is
    that of one state: no field, field along and across the flow, high Lorentz factor, cold."""
    n = (4, 4, 4)
    for v, B, p in ((0.0, (0, 0, 0), 1.0), (0.5, (2.0, 0, 0), 1.0), (0.5, (0, 0.3, 2.0), 0.1), (0.99, (0.1, 0.2, 0.1), 1.0),
                    (0.1, (1.0, 1e-4, 0), 1e-3), (0.0, (3.0, 0, 0), 10.0)):
        P = np.zeros((10, 10, 10, 8))
        P[..., 0], P[..., 1], P[..., 2], P[..., 5:] = 1.0, p, v, B
        ml = {}
        for prec in ("fp64", "fp32"):
            s = Solver(Scheme(precision=prec, extrap="pcm", riemann="hll", advance="single"), n)
            s.upload(P.copy())
            assert s.advance(1e-3) == 0
            ml[prec] = s.max_lambda
        # FP32 states carry 6e-8; the slowest-varying speed of these states amplifies it a
        # thousandfold at the fast = Alfven degeneracy
        assert abs(ml["fp32"] - ml["fp64"]) <= 1e-4, (v, B, p, ml)


@pytest.mark.parametrize("riemann", ["hll", "hllc", "hlld"])
@pytest.mark.parametrize("layout", ["lean", "standard"])
def test_fp32_speeds_of_unequal_sides(riemann, layout):
    """MaxLambda of a step on boxes whose faces have two different states, close (where one side's
    speeds help to start the other's) and far apart, against the restatement."""
    n = (12, 10, 11)
    for P0 in (smooth_box(n, 4), box(n, 4)):
        kw = dict(extrap="plm", riemann=riemann, advance="single")
        cpu, Pc = PortOracle(OScheme(n=n, **kw)), P0.copy()
        assert cpu.advance(Pc, 1e-3) == 0
        s = Solver(Scheme(precision="fp32", layout=layout, **kw), n)
        s.upload(P0.copy())
        assert s.advance(1e-3) == 0
        assert abs(s.max_lambda - cpu.max_lambda) <= 1e-4   # as in the test above
