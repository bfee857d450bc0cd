"""Fields of several megabytes (whole and ragged counts of the copies' pieces) come back from the device
bit for bit through pageable and page-locked memory, also from two threads at once and after the last
context has gone."""

import threading

import numpy as np
import pytest

from tarang_b200 import _lib as L
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu


def round_trip(N, seed, times=3):
    s = IncFluid(N)
    rng = np.random.default_rng(seed)
    for _ in range(times):
        a = rng.standard_normal(s.shape) + 1j * rng.standard_normal(s.shape)
        s.upload(L.TG_WORK0, a)
        assert np.array_equal(s.download(L.TG_WORK0), a)
    s.close()


# 4 MB less and more than the threshold, a whole number of 1 MB pieces, one piece and a bit more, many pieces
@pytest.mark.parametrize("N", [(64, 64, 120), (64, 64, 128), (64, 128, 126), (96, 80, 64), (128, 128, 128)])
def test_round_trip(N):
    round_trip(N, 1)


def test_page_locked():
    import torch
    s = IncFluid((96, 80, 64))
    a = torch.randn(s.shape, dtype=torch.complex128).pin_memory().numpy()
    s.upload(L.TG_WORK0, a)
    assert np.array_equal(s.download(L.TG_WORK0), a)


def test_two_threads():
    err = []

    def run(seed):
        try:
            round_trip((64, 128, 126), seed, 8)
        except BaseException as e:  # noqa: BLE001
            err.append(e)

    t = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not err, err
