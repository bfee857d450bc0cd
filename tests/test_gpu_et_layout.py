"""The energy-transfer products on the eight-lane z-passes (N3 = 128 and 256, dealiased and full
rows): fluxes and shell-to-shell tables against the oracle.  FP64: 1e-12 of the largest entry.
FP32 transforms: an entry is sum_k 2 Re(i k_j P_ij conj R_i) with P_ij = F(H_j G_i), so an error of
2e-6 relative L2 in each P_ij (the transforms' bar) moves it by at most
2 kmax 2e-6 sum_ij |P_ij| |R_i| (Cauchy-Schwarz)."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import _lib as L
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(16, 18, 128), (18, 16, 256)])
@pytest.mark.parametrize("dealias", [True, False])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_transfers(N, dealias, precision):
    V, W = ic.random_phase_field(N, seed=1), ic.random_phase_field(N, k0=3.0, seed=2)
    if dealias:
        V, W = [O.dealias(a) for a in V], [O.dealias(a) for a in W]
    s = IncFluid(N, physics="MHD", nu=2e-3, dt=1e-3, precision=precision, dealias=dealias, n_shells=8)
    s.set_V(V)
    s.set_W(W)
    al = "DEALIAS" if dealias else "ALIAS"
    kf = (1.0, 1.0, 1.0)
    for kind, H, F, R, sign in ((L.TG_ET_UU, V, V, V, -1), (L.TG_ET_UB, W, V, W, 1)):
        f = O.compute_flux_generic(H, F, R, sign, kf, 8, al)
        t = O.compute_shell_tr_generic(H, F, R, sign, kf, 8, al)
        if precision == "FP64":
            tf, tt = 1e-12 * np.abs(f).max(), 1e-12 * np.abs(t).max()
        else:
            h, g = [O.inverse_four(a) for a in H], [O.inverse_four(a) for a in F]
            P = sum(np.linalg.norm(O.forward_four(x * y)) * np.linalg.norm(r) for y, r in zip(g, R) for x in h)
            tf = tt = 2 * O.kmag(N, kf).max() * 2e-6 * P
        assert np.abs(s.Compute_flux(kind) - f).max() < tf
        assert np.abs(s.Compute_shell_tr(kind) - t).max() < tt
