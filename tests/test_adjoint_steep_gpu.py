"""The adjoint on both sides of the aperture from which it adds with atomics (just below 60 degrees),
against the FP64 oracle: a Vrms that rises steeply, padding, ragged tiles, records longer than
the narrow stages."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from poststackmig3d_b200 import Migrator
from poststackmig3d_b200 import synth as S

from helpers import geometry_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angle", [59.0, 60.0, 72.0])
@pytest.mark.parametrize("n_il,n_xl,n_t,pad,amp", [(8, 9, 257, 1, True), (1, 1, 10, 0, True),
                                                   (4, 17, 130, 2, False),
                                                   (3, 5, 5300, 0, True)])
def test_steep_adjoint(n_il, n_xl, n_t, pad, amp, angle):
    W = S.random_workload(7 + n_t, n_il, n_xl, n_t, vel_kind="linear", angle=angle, amp=amp,
                          d_il=15.0, d_xl=12.0, pad_il=pad, pad_xl=pad,
                          dt=0.001 if n_t > 1000 else 0.004)
    v = np.broadcast_to(1500.0 + 2500.0 * np.linspace(0.0, 1.0, n_t), W.data.shape)
    v = np.ascontiguousarray(v, dtype=np.float32)
    W = dataclasses.replace(W, vrms=v)
    g = geometry_for(W)
    im = np.random.default_rng(8).standard_normal((g.n_oi, g.n_ox, g.n_t)).astype(np.float32)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(v)
        got = m.adjoint(im)
    ref = O.adjoint_volume(im.astype(np.float64), v, g.n_il, g.n_xl, g.out_center, g.pad_il,
                           g.pad_xl, g.m_il, np.float32(g.dt_seconds), g.t0(),
                           np.float32(g.tan2), g.d_il, g.d_xl, g.amp, flags=O.CONTRACT)
    rms, mx = rel_err(got, ref)
    assert rms <= 1e-4 and mx <= 1e-4, (rms, mx)  # the operator's FP32 parity bar
