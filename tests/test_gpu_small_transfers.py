"""Whole-array transfers of pageable buffers between 4 and 64 MB, which go as they are for a
solver's first eight and through pinned chunk slots from then on: every one brings the same bytes."""
import numpy as np
import pytest

from ctf_b200 import ics
from ctf_b200.mara import Scheme, Solver

pytestmark = pytest.mark.gpu


# 37^3 guarded zones: below 4 MB; 41 x 42 x 39: just above, three chunks with a short last one;
# 51 x 52 x 50: five; 64^3 guarded zones: whole chunks only
@pytest.mark.parametrize("n", [(31, 31, 31), (35, 36, 33), (45, 46, 44), (58, 58, 58)])
def test_repeated_pageable_transfers_bring_the_same_bytes(n):
    P = ics.turbulence_box(n, seed=3)
    s = Solver(Scheme(), n)
    for k in range(7):   # fourteen transfers
        Q = P * (1.0 + 0.01 * k)
        s.upload(Q.copy())
        assert np.array_equal(s.download(), Q), k
