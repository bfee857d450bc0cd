"""One convection step in the SCFT basis for x lengths around the folded x-pass's row tiles (odd and
even, one to three tiles of 22 or 11 row pairs, an odd number of stored rows) and column counts below
and above one block, against the oracle: 1e-12 (FP64) and 1e-6 (FP32-mixed) relative L2."""

import math

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
KF = (math.pi, math.pi / math.sqrt(2.0), math.pi / math.sqrt(2.0))


def field(rng, N, sine):
    r = rng.standard_normal(N) * np.exp(-np.arange(N[0]) / 6.0)[:, None, None]
    a = O.dealias(np.fft.rfftn(r, axes=(1, 2)) / (N[1] * N[2]), "SCFT")
    if sine:
        a[0] = 0
    return a


@pytest.mark.parametrize("N1", [4, 5, 17, 32, 33, 44, 65, 66, 100, 129])
@pytest.mark.parametrize("N2,N3", [(6, 16), (40, 32)])
@pytest.mark.parametrize("precision,tol", [("FP64", 1e-12), ("FP32", 1e-6)])
def test_step(N1, N2, N3, precision, tol):
    N = (N1, N2, N3)
    rng = np.random.default_rng(N1)
    V = [field(rng, N, i == 0) for i in range(3)]
    p = O.divide_ksqr(O.xderiv(V[0], KF, "SCFT", 1) + O.yderiv(V[1], KF) + O.zderiv(V[2], KF), KF, "SCFT")
    V = [V[0] + O.xderiv(p, KF, "SCFT", 0), V[1] + O.yderiv(p, KF), V[2] + O.zderiv(p, KF)]
    V[0][0] = 0
    T = field(rng, N, True)
    s = IncFluid(N, basis="SCFT", physics="RB", Ra=1e4, Pr=1.0, kfactor=KF, dt=1e-4, precision=precision)
    s.set_V(V)
    s.set_T(T)
    s.step(1)
    u, t, _ = O.RBSolver(N, KF, 1e4, 1.0, 1e-4).step(V, T)
    for g, w in zip(s.get_V() + [s.get_T()], u + [t]):
        assert np.linalg.norm(g - w) <= tol * max(np.linalg.norm(x) for x in u + [t])
