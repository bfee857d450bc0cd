"""A step through the fused stage kernel (k_xstage) gives the bits of the separate passes, for every x length,
physics and precision it takes, with every mode stored, hyper-dissipation, box factors, the RK2 scheme and each force
that reads the stage's fields; so a batch, which takes one or the other by its size, has the bits of a lone run."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import _lib as L
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


def fields(s, physics):
    return s.get_V() + (s.get_W() if physics == "MHD" else []) + ([s.get_T()] if physics == "SCALAR" else [])


def same(a, b):
    return all(np.array_equal(np.asarray(x).view(np.float64), np.asarray(y).view(np.float64)) for x, y in zip(a, b))


OPTIONS = [dict(), dict(dealias=False, scheme="RK2"), dict(hyper_nu=1e-5, kfactor=(1.0, 2.0, 0.5))]
FORCES = [dict(force=dict(inner=1.0, outer=3.0, eps=0.1)), dict(force=dict(kind="coriolis", omega=(0.3, -0.2, 0.5))),
          dict(force=dict(kind="liquid_metal", B0=(0.2, 0.1, 1.0)))]


@pytest.mark.parametrize("N", [(32, 32, 32), (64, 18, 16), (32, 20, 128), (128, 10, 16), (256, 10, 16)])
@pytest.mark.parametrize("physics", ["FLUID", "MHD", "SCALAR"])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_refused_stages(lib, N, physics, precision):
    V, W = (ic.random_phase_field(N, k0=k, seed=i) for i, k in ((1, 4.0), (2, 3.0)))
    for kw in OPTIONS + (FORCES if physics == "FLUID" else FORCES[:1] if physics == "MHD" else []):
        s = IncFluid(N, physics=physics, precision=precision, nu=2e-3, eta=3e-3, kappa=4e-3, dt=1e-3, **kw)
        got = []
        for mask in (0, 2 + 4 + 8 + 128, 4):
            assert lib.tg_debug_set(s.h, L.TG_DEBUG_REFUSE_XSTAGE, mask) == L.TG_OK
            s.set_V(V)
            if physics == "MHD":
                s.set_W(W)
            elif physics == "SCALAR":
                s.set_T(W[0])
            s.step(3)
            got.append(fields(s, physics))
        assert same(got[0], got[1]) and same(got[0], got[2]), kw
        s.close()


# batches within and beyond two waves of tiles (one of the forms with 512 threads)
@pytest.mark.parametrize("N,physics,precision,batch", [
    ((32, 32, 32), "FLUID", "FP64", 16), ((32, 32, 32), "MHD", "FP32", 3), ((32, 32, 32), "MHD", "FP32", 5),
    ((32, 32, 32), "SCALAR", "FP64", 9), ((64, 32, 32), "FLUID", "FP32", 16), ((64, 32, 32), "SCALAR", "FP64", 16),
    ((32, 20, 128), "MHD", "FP64", 8), ((32, 20, 128), "SCALAR", "FP32", 4)])
def test_batch(N, physics, precision, batch):
    from tarang_b200.serving import Server
    n = {"FLUID": 3, "MHD": 6, "SCALAR": 4}[physics]
    cfg = dict(N=N, physics=physics, nu=2e-3, eta=3e-3, kappa=4e-3, dt=1e-3, precision=precision)
    F = [O.dealias(a) for i in (1, 2) for a in ic.random_phase_field(N, k0=3.0, seed=i)][:n]
    s = IncFluid(N, **{k: v for k, v in cfg.items() if k != "N"})
    s.set_V(F[:3])
    if physics == "MHD":
        s.set_W(F[3:])
    elif physics == "SCALAR":
        s.set_T(F[3])
    s.step(3)
    want = fields(s, physics)
    with Server(max_batch=batch) as srv:
        ids = [srv.submit(cfg, F, 3) for _ in range(batch)]
        srv.drain()
        for i in ids:
            assert same(srv.result(i), want)
