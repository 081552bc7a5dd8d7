"""Least-squares migration, resident and sharded, runs one forward operator: the sharded solvers'
slabs give the rows of Migrator.lsm_cg's, bit for bit."""
import numpy as np
import pytest

from poststackmig3d_b200 import Migrator, shard
from poststackmig3d_b200 import synth as S
from poststackmig3d_b200.migration import slab_geometry, split_slabs

from helpers import geometry_for

pytestmark = pytest.mark.gpu


def _scaled_by_one_float(img, p):
    """Whether img is fl(alpha p) for one fp32 alpha (below 2^-120 the kernels flush to zero)."""
    k = np.unravel_index(np.argmax(np.abs(p)), p.shape)
    a = np.float32(img[k] / p[k])
    big = np.abs(img) > 2.0 ** -120
    for step in range(-4, 5):
        c = a
        for _ in range(abs(step)):
            c = np.nextafter(c, np.float32(np.inf if step > 0 else -np.inf), dtype=np.float32)
        if np.array_equal((c * p)[big], img[big]):
            return True
    return False


@pytest.mark.parametrize("n_il,pad_il", [(75, 0), (30, 2)])  # wide and narrow tiles
def test_sharded_forward_is_the_solvers(n_il, pad_il):
    import torch
    W = S.random_workload(9, n_il, 5, 260, vel_kind="lateral", angle=50.0, d_il=14.0, d_xl=11.0,
                          pad_il=pad_il)
    g = geometry_for(W)
    vr = W.vrms_cube()
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms(vr)
        m.set_traces(W.data)
        plain = m.forward()
        img, _ = m.lsm_cg(W.data, 1)  # alpha M d
    assert not _scaled_by_one_float(img, plain)  # the case tells the two orders apart
    for world in (1, 3):
        host, dev = [], []
        for slab in split_slabs(g, world):
            o0, o1, i0, i1 = slab
            lg = slab_geometry(g, slab)
            v = np.ascontiguousarray(vr[i0:i1])
            d = np.ascontiguousarray(W.data[i0:i1])
            ops = shard._SlabOps(lg, v, 0)
            host.append(ops.forward(d))
            ops.close()
            ops = shard._DeviceSlabOps(lg, v, 0)
            with torch.cuda.stream(ops.stream):
                out = ops.forward(torch.from_numpy(d).cuda())
            ops.m.synchronize()
            dev.append(out.cpu().numpy())
            ops.close()
        assert np.array_equal(np.concatenate(host), np.concatenate(dev))
        assert _scaled_by_one_float(img, np.concatenate(host))
