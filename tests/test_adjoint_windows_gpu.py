"""The fp32 adjoint adds into windows that one warp owns at a time, without atomics where the
lanes' addresses are distinct: Vrms fields on both sides of that rule, and edges of the tiles (8
crosslines, 256 samples), against the FP64 oracle."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from poststackmig3d_b200 import Migrator
from poststackmig3d_b200 import synth as S

from helpers import geometry_for, rel_err

pytestmark = pytest.mark.gpu


def _fields(n_il, n_xl, n_t):
    """Vrms fields by name: slopes ds/dt0 around 1, below 1/2 at the aperture's edge, above 1,
    erratic, and with samples that have no Vrms."""
    rng = np.random.default_rng(17)
    t = np.linspace(0.0, 1.0, n_t)
    shape = (n_il, n_xl, n_t)
    holes = np.broadcast_to(2000.0 + 500.0 * t, shape).copy()
    holes[rng.random(shape) < 0.05] = 0.0
    return {"constant": np.full(shape, 2000.0),
            "rising": np.broadcast_to(1000.0 + 5000.0 * t, shape),
            "falling": np.broadcast_to(4000.0 - 2500.0 * t, shape),
            "erratic": rng.uniform(500.0, 5000.0, shape),
            "holes": holes}


@pytest.mark.parametrize("field", ["constant", "rising", "falling", "erratic", "holes"])
@pytest.mark.parametrize("n_il,n_xl,n_t,pad,amp,angle", [
    (9, 11, 300, 1, True, 50.0), (5, 8, 256, 0, False, 70.0), (3, 17, 65, 2, True, 30.0),
    (1, 2, 9, 0, True, 45.0)])
def test_adjoint_over_vrms_fields(field, n_il, n_xl, n_t, pad, amp, angle):
    W = S.random_workload(3 + n_t, n_il, n_xl, n_t, vel_kind="linear", angle=angle, amp=amp,
                          d_il=15.0, d_xl=12.0, pad_il=pad, pad_xl=pad)
    v = np.ascontiguousarray(_fields(n_il, n_xl, n_t)[field], dtype=np.float32)
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


def test_adjoint_leaves_the_record_tail_zero():
    """A trace's stored row ends in zeros; the forward after an adjoint into the ctx's cube reads
    them, so the two calls in a row give the image of the adjoint's own samples."""
    W = S.random_workload(5, 6, 9, 256, vel_kind="linear", angle=60.0)
    g = geometry_for(W)
    im = np.random.default_rng(2).standard_normal((g.n_oi, g.n_ox, g.n_t)).astype(np.float32)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(W.vrms_cube())
        m.set_image(im)
        m.adjoint_async()
        m.synchronize()
        d = m.get_traces()
        m.set_traces(d)  # rewrites the samples, not the rows' tails
        a = m.forward()
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(W.vrms_cube())
        m.set_traces(d)
        assert np.array_equal(a, m.forward())
