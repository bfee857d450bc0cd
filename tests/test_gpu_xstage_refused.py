"""A step whose fused stage kernel (k_xstage) is refused at some stages runs the separate passes there: a forced
fluid (the force reads a band of the stage's fields), a Coriolis force (it reads all of them) and MHD, every mask of
the three stages, against the oracle at 1e-12 (FP64) relative L2.  The kernel's own bounded wait, run out alone, is
reported as TG_ERR_TIMEOUT, and the context runs on afterwards."""

import numpy as np
import pytest

from oracle import tarang_oracle as O
from tarang_b200 import _lib as L
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
KF = (1.0, 1.0, 1.0)


def field(N, k, seed):
    return [O.dealias(a) for a in ic.random_phase_field(N, k0=k, seed=seed)]


@pytest.mark.parametrize("N", [(32, 32, 32), (64, 18, 16)])
@pytest.mark.parametrize("kind", ["band", "coriolis", "mhd"])
def test_masks(lib, N, kind):
    V, W = field(N, 4.0, 1), field(N, 3.0, 2)
    force = dict(band=dict(inner=1.0, outer=3.0, eps=0.1), coriolis=dict(kind="coriolis", omega=(0.3, -0.2, 0.5)),
                 mhd=None)[kind]
    s = IncFluid(N, physics="MHD" if kind == "mhd" else "FLUID", nu=2e-3, eta=3e-3, dt=1e-3, force=force)
    if kind == "mhd":
        m = O.MHDSolver(N, KF, 2e-3, 3e-3, 1e-3)
        u, b, _ = m.step2(V, W)
        u, b, _ = m.step2(u, b)
        want = u + b
    else:
        m = O.FluidSolver(N, KF, 2e-3, 1e-3, force=force)
        want, _ = m.step(m.step(V)[0])
    top = max(np.linalg.norm(x) for x in want)
    for mask in range(8):
        assert lib.tg_debug_set(s.h, L.TG_DEBUG_REFUSE_XSTAGE, 2 * mask) == L.TG_OK  # bits 1, 2, 3
        s.set_V(V)
        if kind == "mhd":
            s.set_W(W)
        s.step(2)
        for g, w in zip(s.get_V() + (s.get_W() if kind == "mhd" else []), want):
            assert np.linalg.norm(g - w) <= 1e-12 * top
    s.close()


def test_own_wait(lib):
    N = (32, 32, 32)
    V = field(N, 4.0, 3)
    s = IncFluid(N, nu=1e-2, dt=1e-3)
    s.set_V(V)
    s.step(1)
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_SHORT_XSTAGE_WAIT, 1) == L.TG_OK
    with pytest.raises(L.TarangError) as ei:
        s.step(2)
    assert ei.value.code == L.TG_ERR_TIMEOUT
    # with every fused stage refused nothing waits short
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_REFUSE_XSTAGE, 14) == L.TG_OK
    s.set_V(V)
    s.step(1)
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_REFUSE_XSTAGE, 0) == L.TG_OK
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_SHORT_XSTAGE_WAIT, 0) == L.TG_OK
    s.set_V(V)
    s.step(1)
    want, _ = O.FluidSolver(N, KF, 1e-2, 1e-3).step(V)
    for g, w in zip(s.get_V(), want):
        assert np.linalg.norm(g - w) <= 1e-12 * max(np.linalg.norm(x) for x in want)
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_SHORT_XSTAGE_WAIT, 2) == L.TG_ERR_ARG
    assert lib.tg_debug_set(s.h, L.TG_DEBUG_REFUSE_XSTAGE, 256) == L.TG_ERR_ARG
    s.close()
