"""Axis passes of lengths that are not powers of two (mixed-radix stages, prime stages, one to four
stages, tiles of eight to two columns) against numpy's FFT, and an MHD step on such a box (the pass
that forms z+ and z-) against the oracle.  Tolerances are the transforms' bars: 1e-13 (FP64), 2e-6
(FP32) relative L2, 1e-12 for a step."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu

LENGTHS = [3, 5, 7, 9, 11, 14, 15, 22, 27, 35, 49, 77, 96, 121, 127, 143, 160, 210, 226, 343, 1001]


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("precision,tol", [("FP64", 1e-13), ("FP32", 2e-6)])
def test_lengths(L, precision, tol):
    rng = np.random.default_rng(L)
    for N in ((L, 6, 8), (4, L, 16)):
        s = IncFluid(N, precision=precision)
        real = rng.standard_normal(N)
        spec = s.Forward_transform_array(O.pack_real(real))
        want = np.fft.rfftn(real) / real.size
        assert np.linalg.norm(spec - want) < tol * np.linalg.norm(want)
        back = O.unpack_real(s.Inverse_transform_array(want))
        assert np.linalg.norm(back - real) < tol * np.linalg.norm(real)
        s.close()


@pytest.mark.parametrize("N", [(22, 18, 16), (48, 26, 32)])
def test_mhd_step(N):
    V, W = ic.random_phase_field(N, seed=1), ic.random_phase_field(N, k0=3.0, seed=2)
    s = IncFluid(N, physics="MHD", nu=2e-3, eta=3e-3, dt=1e-3)
    s.set_V(V)
    s.set_W(W)
    s.step(1)
    u, b, _ = O.MHDSolver(N, (1.0, 1.0, 1.0), 2e-3, 3e-3, 1e-3).step2([O.dealias(a) for a in V], [O.dealias(a) for a in W])
    for g, w in zip(s.get_V() + s.get_W(), u + b):
        assert np.linalg.norm(g - w) < 1e-12 * np.linalg.norm(w)
