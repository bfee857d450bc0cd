"""Axis passes of short lengths that are no power of two, on both sides of the lines between the direct sum and
the mixed-radix stages: lengths of 11 to 29, and column counts around two blocks of eight columns an SM (294 and
301 blocks), against numpy's FFT at the transforms' bars, 1e-13 (FP64) and 2e-6 (FP32) relative L2.  A batch of
requests with such axes gives the bits of a lone run, whichever side a request is on."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [3, 6, 10, 11, 12, 13, 14, 15, 21, 22, 23, 24, 26, 28, 29])
@pytest.mark.parametrize("precision,tol", [("FP64", 1e-13), ("FP32", 2e-6)])
def test_lengths(L, precision, tol):
    rng = np.random.default_rng(L)
    for N in ((L, 48, 96), (L, 49, 96), (3, L, 16)):
        s = IncFluid(N, precision=precision)
        real = rng.standard_normal(N)
        spec = s.Forward_transform_array(O.pack_real(real))
        want = np.fft.rfftn(real) / real.size
        assert np.linalg.norm(spec - want) < tol * np.linalg.norm(want)
        back = O.unpack_real(s.Inverse_transform_array(want))
        assert np.linalg.norm(back - real) < tol * np.linalg.norm(real)
        s.close()


@pytest.mark.parametrize("N", [(12, 14, 16), (26, 10, 32), (14, 96, 64)])
@pytest.mark.parametrize("precision,tol", [("FP64", 1e-12), ("FP32", 1e-6)])
def test_step_and_batch(N, precision, tol):
    from tarang_b200.serving import Server
    cfg = dict(N=N, physics="MHD", nu=2e-3, eta=3e-3, dt=1e-3, precision=precision)
    F = [O.dealias(a) for i in (1, 2) for a in ic.random_phase_field(N, k0=3.0, seed=i)]
    s = IncFluid(N, **{k: v for k, v in cfg.items() if k != "N"})
    s.set_V(F[:3])
    s.set_W(F[3:])
    s.step(1)
    u, b, _ = O.MHDSolver(N, (1.0, 1.0, 1.0), 2e-3, 3e-3, 1e-3).step2(F[:3], F[3:])
    got = s.get_V() + s.get_W()
    for g, w in zip(got, u + b):
        assert np.linalg.norm(g - w) <= tol * max(np.linalg.norm(x) for x in u + b)
    with Server(max_batch=8) as srv:
        ids = [srv.submit(cfg, F, 1) for _ in range(5)]
        srv.drain()
        for i in ids:
            for x, y in zip(srv.result(i), got):
                assert np.array_equal(np.asarray(x).view(np.float64), y.view(np.float64))
