"""Steps on grids whose y-z planes are carried through the y passes and the z-pass in one kernel (k_plane:
N2 and N3 of 32 or 64, with one block a plane and with two), dealiased and with every mode stored, for each
physics, against the oracle: 1e-12 (FP64) and 1e-6 (FP32-mixed) relative L2.  A batch, whose planes take one
block each, gives the bits of a lone run, whose planes take two."""

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


@pytest.mark.parametrize("N", [(6, 32, 32), (48, 32, 64), (50, 64, 32), (74, 64, 64), (96, 64, 64)])
@pytest.mark.parametrize("physics", ["FLUID", "MHD", "SCALAR"])
@pytest.mark.parametrize("dealias", [True, False])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_step(N, physics, dealias, precision):
    V, W = ([O.dealias(a) for a in ic.random_phase_field(N, k0=k, seed=i)] for i, k in ((1, 4.0), (2, 3.0)))
    s = IncFluid(N, physics=physics, nu=2e-3, eta=3e-3, kappa=3e-3, dt=1e-3, precision=precision, dealias=dealias)
    al = "DEALIAS" if dealias else "ALIAS"
    s.set_V(V)
    if physics == "MHD":
        s.set_W(W)
        u, b, _ = O.MHDSolver(N, KF, 2e-3, 3e-3, 1e-3, alias=al).step2(V, W)
        want = u + b
    elif physics == "SCALAR":
        s.set_T(W[0])
        u, t, _ = O.ScalarSolver(N, KF, 2e-3, 3e-3, 1e-3, alias=al).step(V, W[0])
        want = u + [t]
    else:
        want, _ = O.FluidSolver(N, KF, 2e-3, 1e-3, alias=al).step(V)
    s.step(1)
    check(s, want, TOL[precision])


def scft_field(rng, N, sine):
    r = rng.standard_normal(N) * np.exp(-np.arange(N[0]) / 6.0)[:, None, None]
    a = O.dealias(np.fft.rfftn(r, axes=(1, 2)) / (N[1] * N[2]), "SCFT")
    if sine:
        a[0] = 0
    return a


@pytest.mark.parametrize("N", [(9, 32, 32), (49, 32, 64), (96, 64, 32)])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_convection(N, precision):
    kf = (np.pi, np.pi / np.sqrt(2.0), np.pi / np.sqrt(2.0))
    rng = np.random.default_rng(N[0])
    V = [scft_field(rng, N, i == 0) for i in range(3)]
    p = O.divide_ksqr(O.xderiv(V[0], kf, "SCFT", 1) + O.yderiv(V[1], kf) + O.zderiv(V[2], kf), kf, "SCFT")
    V = [V[0] + O.xderiv(p, kf, "SCFT", 0), V[1] + O.yderiv(p, kf), V[2] + O.zderiv(p, kf)]
    V[0][0] = 0
    T = scft_field(rng, N, True)
    s = IncFluid(N, basis="SCFT", physics="RB", Ra=1e4, Pr=1.0, kfactor=kf, dt=1e-4, precision=precision)
    s.set_V(V)
    s.set_T(T)
    s.step(1)
    u, t, _ = O.RBSolver(N, kf, 1e4, 1.0, 1e-4).step(V, T)
    check(s, u + [t], TOL[precision])


@pytest.mark.parametrize("N,physics", [((64, 64, 64), "FLUID"), ((64, 64, 32), "MHD"), ((32, 32, 32), "SCALAR")])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_batch_has_the_bits_of_a_lone_run(N, physics, precision):
    from tarang_b200.serving import Server
    n = {"FLUID": 3, "MHD": 6, "SCALAR": 4}[physics]
    cfg = dict(N=N, physics=physics, nu=2e-3, eta=3e-3, kappa=3e-3, dt=1e-3, precision=precision)
    F = [O.dealias(a) for i in (1, 2) for a in ic.random_phase_field(N, k0=3.0, seed=i)][:n]
    with Server(max_batch=8) as srv:
        ids = [srv.submit(cfg, F, 2) for _ in range(5)]
        srv.drain()
        got = [srv.result(i) for i in ids]
    s = IncFluid(N, **{k: v for k, v in cfg.items() if k != "N"})
    s.set_V(F[:3])
    if n == 6:
        s.set_W(F[3:])
    elif n == 4:
        s.set_T(F[3])
    s.step(2)
    want = s.get_V() + (s.get_W() if n == 6 else []) + ([s.get_T()] if n == 4 else [])
    for g in got:
        for a, b in zip(g, want):
            assert np.array_equal(np.asarray(a).view(np.float64), b.view(np.float64))
