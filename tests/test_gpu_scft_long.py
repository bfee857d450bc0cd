"""One FP64 convection step in the SCFT basis for x lengths whose folded x-pass takes several row blocks, of
each of the row tiles it has (up to the longest x axis), dealiased and with every mode stored, against the
oracle: 1e-12 relative L2."""

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


# MT of the forward / inverse row tiles (of 8 MT row pairs); in brackets with every mode stored, where it differs
@pytest.mark.parametrize("N1", [145,    # 6 / 5
                                257,    # 6 / 9
                                280,    # 6 / 9 [6 / 5]
                                417,    # 3 / 5
                                513,    # 3 / 5 [3 / 2]
                                700,    # 3 / 5 [3 / 2]
                                901,    # 2 / 2
                                1024])  # 2 / 2
@pytest.mark.parametrize("dealias", [True, False])
def test_step(N1, dealias):
    N = (N1, 6, 8)
    rng = np.random.default_rng(N1)
    V = [field(rng, N, i == 0) for i in range(3)]
    p = O.divide_ksqr(O.xderiv(V[0], KF, "SCFT", 1) + O.yderiv(V[1], KF) + O.zderiv(V[2], KF), KF, "SCFT")
    V = [V[0] + O.xderiv(p, KF, "SCFT", 0), V[1] + O.yderiv(p, KF), V[2] + O.zderiv(p, KF)]
    V[0][0] = 0
    T = field(rng, N, True)
    s = IncFluid(N, basis="SCFT", physics="RB", Ra=1e4, Pr=1.0, kfactor=KF, dt=1e-4, dealias=dealias)
    s.set_V(V)
    s.set_T(T)
    s.step(1)
    u, t, _ = O.RBSolver(N, KF, 1e4, 1.0, 1e-4, alias="DEALIAS" if dealias else "ALIAS").step(V, T)
    for g, w in zip(s.get_V() + [s.get_T()], u + [t]):
        assert np.linalg.norm(g - w) <= 1e-12 * max(np.linalg.norm(x) for x in u + [t])
