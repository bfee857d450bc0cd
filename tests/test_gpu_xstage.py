"""Steps whose stages run x-forward, the stage and the next x-inverse in one kernel (k_xstage), for
every x length and physics it takes, both precisions, the RK4 and RK2 schemes, and each force that reads
the stage's fields (a band, a fixed mode, the whole field), two steps against the oracle: 1e-12 (FP64) and
1e-6 (FP32-mixed) relative L2."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
KF = (1.0, 1.0, 1.0)
TOL = {"FP64": 1e-12, "FP32": 1e-6}


def check(s, want, tol):
    got = s.get_V() + (s.get_W() if len(want) == 6 else []) + ([s.get_T()] if len(want) == 4 else [])
    for g, w in zip(got, want):
        assert np.linalg.norm(g - w) <= tol * max(np.linalg.norm(x) for x in want)


@pytest.mark.parametrize("N1", [32, 64, 128, 256])
@pytest.mark.parametrize("physics", ["FLUID", "MHD", "SCALAR"])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_physics(N1, physics, precision):
    N = (N1, 10, 16)
    V, W = ([O.dealias(a) for a in ic.random_phase_field(N, k0=k, seed=i)] for i, k in ((1, 4.0), (2, 3.0)))
    s = IncFluid(N, physics=physics, nu=2e-3, eta=3e-3, kappa=3e-3, dt=1e-3, precision=precision)
    s.set_V(V)
    if physics == "MHD":
        s.set_W(W)
        m = O.MHDSolver(N, KF, 2e-3, 3e-3, 1e-3)
        u, b, _ = m.step2(V, W)
        u, b, _ = m.step2(u, b)
        want = u + b
    elif physics == "SCALAR":
        s.set_T(W[0])
        m = O.ScalarSolver(N, KF, 2e-3, 3e-3, 1e-3)
        u, t, _ = m.step(V, W[0])
        u, t, _ = m.step(u, t)
        want = u + [t]
    else:
        m = O.FluidSolver(N, KF, 2e-3, 1e-3)
        want, _ = m.step(m.step(V)[0])
    s.step(2)
    check(s, want, TOL[precision])


@pytest.mark.parametrize("force", [dict(inner=1.0, outer=3.0, eps=0.1), dict(kind="coriolis", omega=(0.3, -0.2, 0.5)),
                                   dict(kind="liquid_metal", B0=(0.2, 0.1, 1.0))])
@pytest.mark.parametrize("scheme", ["RK4", "RK2"])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_forces(force, scheme, precision):
    N = (32, 18, 32)
    V = [O.dealias(a) for a in ic.random_phase_field(N, seed=5)]
    s = IncFluid(N, nu=2e-3, dt=1e-3, precision=precision, scheme=scheme, force=force)
    s.set_V(V)
    m = O.FluidSolver(N, KF, 2e-3, 1e-3, force=force, scheme=scheme)
    want, _ = m.step(m.step(V)[0])
    s.step(2)
    check(s, want, TOL[precision])
