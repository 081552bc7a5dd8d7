"""The forward kernel at the edges of its tiles (256 samples, 14 or 4 output crosslines), of its
trace windows and of its ring stages, for both kernels and every storage, against the oracle."""
import ctypes
import dataclasses

import numpy as np
import pytest

import oracle as O
from poststackmig3d_b200 import Migrator, _lib
from poststackmig3d_b200 import synth as S
from poststackmig3d_b200._lib import PsmGeom

from helpers import (MAX_REL_TOL, REL_RMS_TOL, dequantized, fp32_floor_ok, geometry_for,
                     oracle_forward, rel_err)

pytestmark = pytest.mark.gpu

WIDE, NARROW = 11, 12


def _images(W, g, variants=(WIDE, NARROW)):
    out = []
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_traces(W.data)
        m.set_vrms(W.vrms_cube())
        for v in variants:
            m.set_variant(v)
            out.append(m.forward())
    return out


@pytest.mark.parametrize("n_il,n_xl,n_t,pad_il,pad_xl", [
    (1, 1, 8, 0, 0), (2, 3, 9, 0, 0), (5, 4, 255, 1, 0), (4, 13, 256, 0, 0),
    (7, 14, 257, 0, 1), (6, 15, 264, 2, 3), (3, 29, 33, 0, 0), (9, 5, 513, 0, 2),
    (33, 20, 100, 1, 1)])
def test_tile_edges_match_the_oracle(n_il, n_xl, n_t, pad_il, pad_xl):
    W = S.random_workload(61 + n_t, n_il, n_xl, n_t, vel_kind="lateral", angle=50.0, d_il=12.0,
                          d_xl=9.0, pad_il=pad_il, pad_xl=pad_xl)
    g = geometry_for(W)
    ref, _, _ = oracle_forward(W, g)
    for img in _images(W, g):
        rms, mx = rel_err(img, ref)
        assert rms <= REL_RMS_TOL and mx <= MAX_REL_TOL, (rms, mx)
        assert np.array_equal(img == 0, ref == 0)


@pytest.mark.parametrize("precision,compensated", [("f32", False), ("f32", True),
                                                   ("bf16", False), ("f16", True)])
def test_windows_longer_than_a_stage(precision, compensated):
    """Vrms between 300 and 6000 m/s from sample to sample: a trace's window covers nearly all
    of its 5200 samples, more than a ring stage of either kernel holds, and is staged in
    parts."""
    rng = np.random.default_rng(5)
    n_il, n_xl, n_t = 4, 6, 5200
    W = S.random_workload(71, n_il, n_xl, n_t, vel_kind="linear", angle=60.0, dt=0.001,
                          d_il=40.0, d_xl=30.0)
    W = dataclasses.replace(W, vrms=rng.uniform(300.0, 6000.0, W.data.shape).astype(np.float32))
    g = dataclasses.replace(geometry_for(W), precision=precision, compensated=compensated)
    Wq = dataclasses.replace(W, data=dequantized(W.data, precision)) if precision != "f32" else W
    ref, _, _ = oracle_forward(Wq, g)
    _, ref64, _ = oracle_forward(Wq, g, O.CONTRACT | O.F64, want64=True)
    variants = (WIDE, NARROW)
    for img in _images(W, g, variants):
        ok, errs = fp32_floor_ok(img, ref, ref64)
        assert ok, errs


def test_a_trace_with_infinities_stays_alone():
    """Windows of several traces lie side by side in a stage: non-finite samples of one trace
    reach only the output samples that sum it, as in a migration without its neighbours."""
    W = S.random_workload(81, 5, 9, 120, vel_kind="linear", angle=20.0, d_il=60.0, d_xl=60.0)
    bad = W.data.copy()
    bad[2, 4, 50:] = np.inf
    bad[1, 7] = np.nan
    g = geometry_for(W)
    only = np.zeros_like(W.data)
    only[2, 4, 49:] = 1.0  # (sample 49's difference is infinite too)
    only[1, 7] = 1.0
    touched = [i != 0 for i in _images(dataclasses.replace(W, data=only), g)]
    clean = _images(W, g)
    for img, ref, t in zip(_images(dataclasses.replace(W, data=bad), g), clean, touched):
        assert np.array_equal(img[~t], ref[~t])
        assert not np.isfinite(img[t]).all()


@pytest.mark.parametrize("n_t", [264, 250])
def test_noalloc_pairs_of_whole_rows(n_t):
    """Rows of exactly n_t pairs (n_t a multiple of 8) end where a window may end: the same
    image as the resident forward, whose rows have a zero tail."""
    import torch
    W = S.random_workload(91, 8, 16, n_t, vel_kind="lateral", pad_il=1, pad_xl=2)
    g = geometry_for(W)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_traces(W.data)
        m.set_vrms(W.vrms_cube())
        ref = m.forward()
    ns = (n_t + 7) & ~7
    d = torch.zeros((8, 16, ns + 1), device="cuda")
    d[..., :n_t] = torch.from_numpy(W.data).cuda()
    pairs = torch.stack([d[..., :ns], d[..., 1:] - d[..., :ns]], dim=-1).contiguous()
    vr = torch.from_numpy(W.vrms_cube()).cuda()
    img = torch.full(ref.shape, float("nan"), device="cuda")
    torch.cuda.synchronize()
    f = _lib.cuda().psm_forward_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.POINTER(PsmGeom)] + [ctypes.c_void_p] * 5
    gc = g.to_c()
    assert f(ctypes.byref(gc), None, pairs.data_ptr(), vr.data_ptr(), img.data_ptr(), None) == 0
    assert np.array_equal(img.cpu().numpy(), ref)


def test_solver_operator_equals_forward():
    """The least-squares operator adds terms in trace order: with no iteration the residual is
    the data, and one iteration follows alpha = |M d|^2 / |M^T M d|^2 with the forward's image
    to FP32 rounding."""
    W = S.random_workload(95, 11, 17, 270, vel_kind="lateral", pad_il=1)
    g = geometry_for(W)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(W.vrms_cube())
        m.set_traces(W.data)
        img = m.forward().astype(np.float64)
        q = m.adjoint(img.astype(np.float32)).astype(np.float64)
        got, hist = m.lsm_cg(W.data, 1)
    alpha = float((img ** 2).sum() / (q ** 2).sum())
    assert abs(hist[0] - np.linalg.norm(W.data.astype(np.float64))) <= 1e-6 * hist[0]
    assert rel_err(got, alpha * img)[0] <= 1e-5
