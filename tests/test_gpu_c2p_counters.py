"""The counters of an advance: the c2p outcomes on a box whose neighbouring zones -- lanes of one warp
-- resolve on different rungs of the ladder, against the C restatement zone by zone, and the faces of the lean sweeps, each counted once."""
import numpy as np
import pytest

from ctf_b200 import ics
from ctf_b200.mara import Scheme, Solver
from oracle import PortOracle, Scheme as OScheme

pytestmark = pytest.mark.gpu


def rung_of(port, U, guess):
    """The rung on which the ladder resolves U from the previous primitives `guess` (0: none),
    and its primitives."""
    for rung, (solver, start) in enumerate(((0, 0), (0, 1), (1, 0), (1, 1)), 1):
        P, e, _ = port.c2p_solve(U, solver, start, guess)
        if e == 0:
            return rung, P
    return 0, None


def mixed_zones(golden, port):
    """Primitives that a first c2p (previous primitives zero) resolves, and their rungs in that
    c2p and in the next."""
    rows = []
    for P in np.concatenate([golden("c2p_paths.npz")["P_ladder"], golden("c2p.npz")["P"][:100]]):
        U, e = port.prim_to_cons(P)
        if e or not np.isfinite(U).all():
            continue
        first, Q = rung_of(port, U, np.zeros(8))
        if first:
            rows.append((P, first, rung_of(port, U, Q)[0]))
    return rows


def test_outcomes_of_a_warp_are_counted_each_on_its_own_rung(golden):
    """With emergency resets on, one zone in ten has a conserved state that fails its checks before
    any rung: it counts as a failed call and on no rung."""
    n = (8, 8, 8)
    port = PortOracle(OScheme(n=n))
    rows = mixed_zones(golden, port)
    rng = np.random.default_rng(1)
    pick, bad = rng.integers(0, len(rows), 512), rng.random(512) < 0.1
    inner = np.array([rows[k][0] for k in pick])
    inner[bad] = (1.0, -1.0, 0, 0, 0, 0, 0, 0)
    s = Solver(Scheme(extrap="pcm", riemann="hll", advance="single", ereset=True), n)
    s.upload(ics.with_guards(np.ascontiguousarray(inner.reshape(n + (8,)))))
    s.advance(0.0)                                           # U stays: two c2p of it per zone
    want = [0] * 6
    for k in pick[~bad]:
        want[rows[k][1]] += 1
        want[rows[k][2]] += 1
    assert sum(w > 0 for w in want) >= 3                     # rung 1 and two others at least
    st = s.stats()
    assert st["c2p_calls"] == 2 * 512 and st["c2p_failed"] == 2 * bad.sum()
    assert list(st["c2p_attempt"]) == want


@pytest.mark.parametrize("precision,extrap", [("fp32", "plm"), ("fp32", "weno5"), ("fp64", "plm")])
@pytest.mark.parametrize("n", [(9, 17, 33), (47, 12, 130), (20, 64, 5)])
def test_lean_sweeps_count_each_face_once(n, precision, extrap):
    """A chunk of a marching sweep, and a block of the z sweep, solves its first face again; short
    chunks repeat up to one face in three."""
    s = Solver(Scheme(precision=precision, layout="lean", extrap=extrap, advance="rk2"), n)
    s.upload(ics.turbulence_box(n, seed=2))
    assert s.advance(1e-4) == 0
    st = s.stats()
    faces = sum((n[d] + 1) * (n[(d + 1) % 3] + 2) * (n[(d + 2) % 3] + 2) for d in range(3))
    assert st["hlld_ok"] + st["hlld_hllc"] == 2 * faces
