"""psm_forward_noalloc in wide tiles: the mirrors of caller-made pairs go through one buffer for all
ring stages, and the image is the resident forward's bit for bit."""
import ctypes
import dataclasses

import numpy as np
import pytest

from poststackmig3d_b200 import Migrator, _lib
from poststackmig3d_b200 import synth as S
from poststackmig3d_b200._lib import PsmGeom

from helpers import geometry_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_il,n_xl,n_t,steep", [
    (40, 30, 264, False),    # many stages a tile, pairs and single traces; rows of n_t pairs
    (90, 15, 250, False),
    (5, 15, 4800, True)])    # windows longer than a stage, staged in parts
def test_wide_noalloc_equals_resident_forward(n_il, n_xl, n_t, steep):
    import torch
    W = S.random_workload(n_t, n_il, n_xl, n_t, vel_kind="linear", angle=50.0, d_il=15.0,
                          d_xl=12.0, dt=0.001 if steep else 0.004)
    if steep:
        v = np.random.default_rng(3).uniform(300.0, 6000.0, W.data.shape).astype(np.float32)
        W = dataclasses.replace(W, vrms=v)
    g = geometry_for(W)
    assert g.n_oi * -(-g.n_ox // 14) * -(-n_t // 256) >= 148  # wide by default
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_traces(W.data)
        m.set_vrms(W.vrms_cube())
        ref = m.forward()
    ns = (n_t + 7) & ~7
    d = torch.zeros((n_il, n_xl, ns + 1), device="cuda")
    d[..., :n_t] = torch.from_numpy(W.data).cuda()
    pairs = torch.stack([d[..., :ns], d[..., 1:] - d[..., :ns]], dim=-1).contiguous()
    vr = torch.from_numpy(W.vrms_cube()).cuda()
    img = torch.full(ref.shape, float("nan"), device="cuda")
    torch.cuda.synchronize()
    f = _lib.cuda().psm_forward_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.POINTER(PsmGeom)] + [ctypes.c_void_p] * 5
    gc = g.to_c()
    oc = np.ascontiguousarray(g.out_center, dtype=np.int32)
    for _ in range(3):
        assert f(ctypes.byref(gc), oc.ctypes.data, pairs.data_ptr(), vr.data_ptr(),
                 img.data_ptr(), None) == 0
        assert np.array_equal(img.cpu().numpy(), ref)
        img.fill_(float("nan"))
        torch.cuda.synchronize()
