"""Field copies of a context that has moved enough for the copying threads to have been set up: whole and ragged
counts of their pieces, from one thread and from two, come back from the device bit for bit."""

import threading

import numpy as np
import pytest

from tarang_b200 import _lib as L
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def owner():
    s = IncFluid((256, 128, 128))
    a = np.zeros(s.shape, np.complex128)
    for _ in range(5):  # 34 MB each
        s.upload(L.TG_WORK0, a)
    yield s
    s.close()


@pytest.mark.parametrize("N", [(64, 64, 120), (64, 64, 128), (64, 128, 126), (96, 80, 64), (128, 128, 128)])
def test_round_trip(owner, N):
    err = []

    def run(seed):
        try:
            s = IncFluid(N)
            rng = np.random.default_rng(seed)
            for _ in range(4):
                a = rng.standard_normal(s.shape) + 1j * rng.standard_normal(s.shape)
                s.upload(L.TG_WORK0, a)
                assert np.array_equal(s.download(L.TG_WORK0), a)
            s.close()
        except BaseException as e:  # noqa: BLE001
            err.append(e)

    run(0)
    t = [threading.Thread(target=run, args=(i,)) for i in (1, 2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not err, err
