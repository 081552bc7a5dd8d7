"""psm_kirchhoff_inline takes the caller's output times in any order: the forward kernel's trace
windows cover the terms of every sample of a tile, and the image is the oracle's sample for
sample (each output sample depends on its own t0 only)."""
import numpy as np
import pytest

import oracle as O
from poststackmig3d_b200 import MigrationKernel

from helpers import MAX_REL_TOL, REL_RMS_TOL, rel_err

pytestmark = pytest.mark.gpu


def _orders(n_t, dt):
    t0 = O.t0_times(n_t, dt)
    rng = np.random.default_rng(n_t)
    holes = t0.copy()
    holes[::7] = 0.0
    holes[3::11] = -1.0
    return {"reversed": t0[::-1].copy(), "shuffled": rng.permutation(t0),
            "by threes": np.concatenate([t0[k::3] for k in range(3)]), "holes": holes}


@pytest.mark.parametrize("order", ["reversed", "shuffled", "by threes", "holes"])
@pytest.mark.parametrize("n_il,n_xl,n_t,n_out,dt", [
    (9, 14, 150, 20, 0.004),    # narrow tiles, a window within a stage
    (3, 5, 2900, 7, 0.002),     # narrow tiles, windows longer than a stage (2432 samples)
    (3, 40, 3840, 130, 0.001)])  # wide tiles (10 x 15 of them)
def test_any_order_of_output_times(n_il, n_xl, n_t, n_out, dt, order):
    rng = np.random.default_rng(n_xl)
    buf = rng.standard_normal((n_il, n_xl, n_t)).astype(np.float32)
    vel = (1800 + 400 * rng.random((n_xl, n_t))).astype(np.float32)
    il_pos = np.arange(n_il, dtype=np.int32)
    t0 = _orders(n_t, dt)[order]
    tan2 = O.tan2_theta(35.0)
    out = np.full((n_out, n_t), np.nan, dtype=np.float32)
    MigrationKernel.kirchhoff_kernel_3d_with_padding(
        buf, n_il, n_xl, n_t, vel, out, il_pos, None, n_il // 2, -2, dt, t0, tan2, 25.0, 20.0,
        True)
    ref, _, _ = O.kirchhoff_inline(buf, vel, n_out, il_pos, n_il // 2, -2, dt, t0, tan2, 25.0,
                                   20.0, True)
    rms, mx = rel_err(out, ref)
    assert rms <= REL_RMS_TOL and mx <= MAX_REL_TOL, (rms, mx)
    assert np.array_equal(out == 0, ref == 0)
