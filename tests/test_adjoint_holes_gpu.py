"""The adjoint where samples have no Vrms: they spread nothing, and the samples around them still go
through the windows without atomics; holes at the ends and in the middle of lanes (2 samples),
blocks (64) and warps (256), against the FP64 oracle."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from poststackmig3d_b200 import Migrator
from poststackmig3d_b200 import synth as S

from helpers import geometry_for, rel_err

pytestmark = pytest.mark.gpu

N_T = 333
HOLES = {"even": np.arange(N_T) % 2 == 0, "odd": np.arange(N_T) % 2 == 1,
         "sparse": np.arange(N_T) % 97 == 5, "pairs": np.arange(N_T) % 6 < 2,
         "block": (np.arange(N_T) >= 64) & (np.arange(N_T) < 128),
         "top": np.arange(N_T) < 70, "bottom": np.arange(N_T) >= 250,
         "tile": np.arange(N_T) < 256, "all but one": np.arange(N_T) != 131}


@pytest.mark.parametrize("name", list(HOLES))
@pytest.mark.parametrize("rising", [False, True])
def test_adjoint_with_holes(name, rising):
    W = S.random_workload(21, 7, 10, N_T, vel_kind="linear", angle=40.0, d_il=15.0, d_xl=12.0,
                          pad_il=1)
    t = np.linspace(0.0, 1.0, N_T)
    v = np.broadcast_to(1600.0 + (1500.0 if rising else 0.0) * t, W.data.shape)
    v = v.astype(np.float32)
    v[:, ::2, HOLES[name]] = 0.0  # (every other crossline is whole)
    v[3, 5, HOLES[name]] = 1e-6
    W = dataclasses.replace(W, vrms=v)
    g = geometry_for(W)
    im = np.random.default_rng(4).standard_normal((g.n_oi, g.n_ox, g.n_t)).astype(np.float32)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(v)
        got = m.adjoint(im)
    ref = O.adjoint_volume(im.astype(np.float64), v, g.n_il, g.n_xl, g.out_center, g.pad_il,
                           g.pad_xl, g.m_il, np.float32(g.dt_seconds), g.t0(),
                           np.float32(g.tan2), g.d_il, g.d_xl, g.amp, flags=O.CONTRACT)
    rms, mx = rel_err(got, ref)
    assert rms <= 1e-4 and mx <= 1e-4, (rms, mx)  # the operator's FP32 parity bar
