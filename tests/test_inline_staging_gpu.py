"""psm_kirchhoff_inline copies directly on a thread's first call and through its pinned staging
buffers (3 of 2 MB, rows at the device's pitch) from the second on: the same bits."""
import threading

import numpy as np
import pytest

from poststackmig3d_b200 import MigrationKernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_il,n_xl,n_t", [(3, 5, 7), (3, 5, 8), (11, 40, 1193), (17, 61, 2003)])
def test_staged_calls_equal_the_first(n_il, n_xl, n_t):
    rng = np.random.default_rng(n_t)
    vel = (1800 + 400 * rng.random((n_xl, n_t))).astype(np.float32)
    il_pos = np.arange(n_il, dtype=np.int32)
    t0 = (np.arange(n_t) * 0.004).astype(np.float32)
    bufs = [rng.standard_normal((n_il, n_xl, n_t)).astype(np.float32) for _ in range(2)]

    def call(buf):
        out = np.full((n_xl + 2, n_t), np.nan, dtype=np.float32)
        MigrationKernel.kirchhoff_kernel_3d_with_padding(
            buf, n_il, n_xl, n_t, vel, out, il_pos, None, n_il // 2, -1, 0.004, t0, 0.5, 25.0,
            20.0, True)
        return out

    got = {}

    def run(first):  # a thread of its own: its first call is direct, the others staged
        got[first] = [call(bufs[first]), call(bufs[1 - first]), call(bufs[first])]

    for first in (0, 1):
        t = threading.Thread(target=run, args=(first,))
        t.start()
        t.join()
    for first in (0, 1):
        direct, other, again = got[first]
        assert np.isfinite(direct).all()
        assert np.array_equal(direct, again)
        assert np.array_equal(other, got[1 - first][0])
