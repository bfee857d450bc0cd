"""One step on grids whose z rows are short (N3 = 8 .. 64, k_z_prod_rows), with row counts that leave
the last block part empty, against the oracle: 1e-12 (FP64) and 1e-6 (FP32-mixed) relative L2."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
KF = (1.0, 1.0, 1.0)


@pytest.mark.parametrize("N", [(6, 10, 8), (10, 7, 16), (6, 14, 32), (10, 9, 64)])
@pytest.mark.parametrize("physics", ["FLUID", "MHD", "SCALAR"])
@pytest.mark.parametrize("precision,tol", [("FP64", 1e-12), ("FP32", 1e-6)])
def test_step(N, physics, precision, tol):
    V, W = ([O.dealias(a) for a in ic.random_phase_field(N, k0=k, seed=i)] for i, k in ((1, 4.0), (2, 3.0)))
    s = IncFluid(N, physics=physics, nu=2e-3, eta=3e-3, kappa=3e-3, dt=1e-3, precision=precision)
    s.set_V(V)
    if physics == "MHD":
        s.set_W(W)
        u, b, _ = O.MHDSolver(N, KF, 2e-3, 3e-3, 1e-3).step2(V, W)
        want = u + b
    elif physics == "SCALAR":
        s.set_T(W[0])
        u, t, _ = O.ScalarSolver(N, KF, 2e-3, 3e-3, 1e-3).step(V, W[0])
        want = u + [t]
    else:
        want, _ = O.FluidSolver(N, KF, 2e-3, 1e-3).step(V)
    s.step(1)
    got = s.get_V() + (s.get_W() if physics == "MHD" else []) + ([s.get_T()] if physics == "SCALAR" else [])
    for g, w in zip(got, want):
        assert np.linalg.norm(g - w) <= tol * max(np.linalg.norm(x) for x in want)
