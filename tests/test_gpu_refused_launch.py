"""A call that is refused by a launch (a sine/cosine transform whose tables exceed the shared memory) fails by
itself only: the next calls, on that context and on another, run and give the right values."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import _lib as L
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


def test_error_does_not_reach_the_next_call():
    N = (32, 32, 32)
    V = [O.dealias(a) for a in ic.random_phase_field(N, seed=4)]
    s = IncFluid(N, nu=1e-2, n_shells=8)
    s.set_V(V)
    want = s.CV_Compute_shell_spectrum()
    r = IncFluid((513, 4, 8), basis="SCFT", physics="RB", Ra=1e4, Pr=1.0)

    def refused():
        with pytest.raises(L.TarangError):
            r.Forward_transform_array(np.zeros(r.shape, np.complex128))

    refused()
    for a, b in zip(s.CV_Compute_shell_spectrum(), want):
        assert np.array_equal(a, b)
    refused()
    r.step(1)
    s.step(1)
    ref, _ = O.FluidSolver(N, (1.0, 1.0, 1.0), 1e-2, s.cfg.dt).step(V)
    for a, b in zip(s.get_V(), ref):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    s.close()
    r.close()
