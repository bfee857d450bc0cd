"""Downloads of several megabytes into fresh pageable memory on a stream of the caller's, ordinary or the
per-thread default one, right behind the work that fills the field: a transform of a work field and a state
field after a step, with the bits of a context on a stream of its own."""

import numpy as np
import pytest

from tarang_b200 import _lib as L
from tarang_b200 import ic
from tarang_b200.solver import IncFluid

pytestmark = pytest.mark.gpu
N = (128, 128, 128)
PER_THREAD = 2  # cudaStreamPerThread


@pytest.mark.parametrize("kind", ["ordinary", "per-thread"])
def test_downloads(kind):
    import torch
    stream = torch.cuda.Stream() if kind == "ordinary" else None
    a, b = IncFluid(N, nu=1e-2), IncFluid(N, nu=1e-2, stream=stream.cuda_stream if stream else PER_THREAD)
    rng = np.random.default_rng(1)
    real = np.zeros((N[0], N[1], N[2] + 2))
    real[:, :, : N[2]] = rng.standard_normal(N)
    for k in range(8):
        packed = np.ascontiguousarray(np.roll(real, k, axis=0)).view(np.complex128)
        want = a.Forward_transform_array(packed)
        assert np.array_equal(b.Forward_transform_array(packed), want)
        assert np.array_equal(b.Inverse_transform_array(want), a.Inverse_transform_array(want))
    V = ic.random_phase_field(N, seed=3)
    for s in (a, b):
        s.set_V(V)
        s.step(1)
    for k in range(3):
        assert np.array_equal(b.download(L.TG_V1 + k), a.download(L.TG_V1 + k))
    a.close()
    b.close()
