"""The faces of test_faces_host.py through the device's FP64 HLLD, against the C restatement."""
import numpy as np
import pytest

from tests.test_faces_host import MEETING, face_rel, oracle_hlld, random_faces
from tests.test_gpu_functions import RIEMANN_REL, probe_riemann

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wmax", [10.0, 50.0])
def test_relativistic_jumps_fall_back_to_hllc_where_the_oracle_does(wmax):
    P, Q = random_faces(3000, wmax, 0.5)
    P, Q = np.concatenate([MEETING[0], P]), np.concatenate([MEETING[1], Q])
    F0, e0, u0 = oracle_hlld(P, Q)
    # CUDA's libm moves the wave speeds by an ulp or two: leave out the faces on which the
    # restatement itself changes branch, or its flux, when its libm is off by as much
    F1, e1, u1 = oracle_hlld(P, Q, perturbed_libm=True)
    firm = (u0 == u1) & (e0 == 0) & (e1 == 0)
    firm[firm] = face_rel(F1[firm], F0[firm]) <= RIEMANN_REL
    assert firm[0] and firm.mean() > 0.95, firm.mean()
    F, e, _, u = probe_riemann(2, P, Q, 1)
    assert not e[firm].any()
    assert np.array_equal(u[firm] != 0, u0[firm])
    # the device's ulp and the perturbed restatement's need not be the same: twice the bound
    assert face_rel(F[firm], F0[firm]).max() <= 2 * RIEMANN_REL
