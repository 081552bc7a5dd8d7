"""Calls that return an image report the kernels' error word: it is zero until a kernel sets it,
also when no kernel has run since the geometry was set and the device memory held something
else before."""
import numpy as np
import pytest

from poststackmig3d_b200 import Batch, Migrator, Problem
from poststackmig3d_b200 import synth as S

from helpers import geometry_for

pytestmark = pytest.mark.gpu


def _leave_garbage(W, g):
    """A context whose small buffers held other values is gone: its memory is handed out again."""
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(W.vrms_cube())
        m.set_traces(W.data)
        m.set_image(np.full(m.image_shape(), 3.0e7, dtype=np.float32))


@pytest.mark.parametrize("n_t", [9, 60, 127])
def test_image_that_no_kernel_wrote(n_t):
    W = S.random_workload(n_t, 4, 5, n_t, vel_kind="linear")
    g = geometry_for(W)
    with Migrator(0) as first:  # (keeps the driver's blocks of small allocations)
        first.set_geometry(g)
        for _ in range(4):
            _leave_garbage(W, g)
            with Migrator(0) as m:
                m.set_geometry(g)
                img = np.arange(np.prod(m.image_shape()), dtype=np.float32).reshape(
                    m.image_shape())
                m.set_image(img)
                assert np.array_equal(m.get_image(), img)
            _leave_garbage(W, g)
            with Migrator(0) as m, Batch(m, [Problem(g, W.data, W.vrms_cube())]) as b:
                b.image(0)
