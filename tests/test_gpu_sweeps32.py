"""The FP32 sweeps at the sizes where their tiling can go wrong, against the FP64 restatement:
rows shorter and longer than a block of the z sweep (126 zones per block), the smallest box,
columns that do not fill a block, every reconstruction; and face states the fast-speed
iteration must hand to the closed form.  Bounds: those of the FP32-bulk path
(test_gpu_fp32.py), which one step of a random box stays a hundred times below."""
import numpy as np
import pytest

from ctf_b200 import ics
from ctf_b200.mara import Scheme, Solver
from oracle import PortOracle, Scheme as OScheme
from tests.test_gpu_fp32 import L1_TOL, LINF_TOL, rel_errors

pytestmark = pytest.mark.gpu


def box(n, seed):
    """Turbulence with density and pressure fluctuations (every component varies)."""
    rng = np.random.default_rng(seed)
    P = ics.turbulence_box(n, seed=seed, vrms=0.3)
    inner = P[3:-3, 3:-3, 3:-3]
    inner[..., :2] = np.exp(0.1 * rng.standard_normal(inner.shape[:3] + (2,)))
    return ics.with_guards(np.ascontiguousarray(inner))


@pytest.mark.parametrize("extrap", ["pcm", "plm", "weno5"])
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 3, 126), (3, 5, 125), (9, 17, 33), (35, 6, 4)])
def test_fp32_hlld_sweeps_match_the_oracle(n, extrap):
    kw = dict(extrap=extrap, riemann="hlld", advance="rk2")
    P0 = box(n, 5)
    cpu, Pc = PortOracle(OScheme(n=n, **kw)), P0.copy()
    dt = 0.1 / max(n)
    assert cpu.advance(Pc, dt) == 0
    for layout in ("lean", "standard"):
        s = Solver(Scheme(precision="fp32", layout=layout, **kw), n)
        s.upload(P0.copy())
        assert s.advance(dt) == 0
        l1, linf = rel_errors(s.download(), Pc, 3)
        assert l1.max() <= L1_TOL and linf.max() <= LINF_TOL, (layout, l1, linf)
        st = s.stats()
        assert st["hlld_hllc"] <= 0.01 * st["hlld_ok"]


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
