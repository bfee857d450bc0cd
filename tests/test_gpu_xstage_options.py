"""Steps through k_xstage with every mode stored, box factors other than one and hyper-dissipation, and FP32 MHD and
scalar grids on both sides of its line (one wave of tiles), against the oracle: 1e-12 (FP64) and 1e-6 (FP32-mixed)
relative L2."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
TOL = {"FP64": 1e-12, "FP32": 1e-6}


def compare(N, physics, precision, dealias=True, kf=(1.0, 1.0, 1.0), hyper=0.0, n=2):
    V, W = ([O.dealias(a) for a in ic.random_phase_field(N, k0=k, seed=i)] for i, k in ((1, 4.0), (2, 3.0)))
    s = IncFluid(N, physics=physics, nu=2e-3, eta=3e-3, kappa=3e-3, dt=1e-3, precision=precision, dealias=dealias,
                 kfactor=kf, hyper_nu=hyper)
    al = "DEALIAS" if dealias else "ALIAS"
    s.set_V(V)
    if physics == "MHD":
        s.set_W(W)
        m = O.MHDSolver(N, kf, 2e-3, 3e-3, 1e-3, alias=al, nu_h=hyper, eta_h=hyper)
        u, b = V, W
        for _ in range(n):
            u, b, _ = m.step2(u, b)
        want = u + b
    elif physics == "SCALAR":
        s.set_T(W[0])
        m = O.ScalarSolver(N, kf, 2e-3, 3e-3, 1e-3, alias=al, nu_h=hyper, kappa_h=hyper)
        u, t = V, W[0]
        for _ in range(n):
            u, t, _ = m.step(u, t)
        want = u + [t]
    else:
        m = O.FluidSolver(N, kf, 2e-3, 1e-3, alias=al, nu_h=hyper)
        want = V
        for _ in range(n):
            want, _ = m.step(want)
    s.step(n)
    got = s.get_V() + (s.get_W() if physics == "MHD" else []) + ([s.get_T()] if physics == "SCALAR" else [])
    top = max(np.linalg.norm(x) for x in want)
    for g, w in zip(got, want):
        assert np.linalg.norm(g - w) <= TOL[precision] * top


@pytest.mark.parametrize("N1,physics,precision", [(32, "FLUID", "FP32"), (32, "MHD", "FP64"), (64, "SCALAR", "FP64"),
                                                  (64, "MHD", "FP32"), (128, "FLUID", "FP64"), (256, "FLUID", "FP64")])
@pytest.mark.parametrize("option", [dict(dealias=False), dict(hyper=1e-5), dict(kf=(1.0, 2.0, 0.5)),
                                    dict(dealias=False, hyper=1e-5, kf=(0.5, 1.0, 1.5))])
def test_options(N1, physics, precision, option):
    compare((N1, 10, 16), physics, precision, **option)


# tiles of eight columns: 147 (fused), 150 and 297 (the separate passes)
@pytest.mark.parametrize("N2", [76, 78, 152])
@pytest.mark.parametrize("physics", ["MHD", "SCALAR"])
def test_lines(N2, physics):
    compare((32, N2, 64), physics, "FP32", n=1)
