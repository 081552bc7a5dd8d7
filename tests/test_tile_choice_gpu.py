"""The tiles that the default variant takes: which of the two kernels a problem runs, told by its
image bit for bit (the two add an output sample's terms in different orders)."""
import dataclasses

import numpy as np
import pytest

from poststackmig3d_b200 import Batch, Migrator, Problem
from poststackmig3d_b200 import synth as S
from poststackmig3d_b200.shard import migrate_shard

from helpers import geometry_for

pytestmark = pytest.mark.gpu

DEFAULT, WIDE, NARROW = 0, 11, 12


def _workload(n_il, n_xl, n_t, pad_xl=0, seed=5):
    return S.random_workload(seed, n_il, n_xl, n_t, vel_kind="lateral", angle=50.0, d_il=14.0,
                             d_xl=11.0, pad_xl=pad_xl)


def _context(m, W, g):
    m.set_geometry(g)
    m.set_traces(W.data)
    m.set_vrms(W.vrms_cube())


def _images(W, g):
    with Migrator(0) as m:
        _context(m, W, g)
        out = {}
        for v in (DEFAULT, WIDE, NARROW):
            m.set_variant(v)
            out[v] = m.forward()
    assert not np.array_equal(out[WIDE], out[NARROW])  # the case tells them apart
    return out


@pytest.mark.parametrize("n_il,n_xl,n_t,pad_xl,narrow", [
    (90, 2, 260, 1, True), (90, 3, 260, 1, False),  # 4 and 5 output crosslines
    (73, 5, 260, 0, True), (74, 5, 260, 0, False)])  # 146 and 148 wide tiles
def test_default_tiles(n_il, n_xl, n_t, pad_xl, narrow):
    W = _workload(n_il, n_xl, n_t, pad_xl)
    img = _images(W, geometry_for(W))
    assert np.array_equal(img[DEFAULT], img[NARROW if narrow else WIDE])


@pytest.mark.parametrize("n_il,narrow", [(73, True), (74, False)])
@pytest.mark.parametrize("precision,compensated", [("f32", False), ("f32", True), ("bf16", False)])
def test_reported_variant_is_the_one_that_runs(n_il, narrow, precision, compensated):
    """The default's id is that of its tiles, and setting it gives the same image; id 13 runs the
    narrow tiles with every storage and sum."""
    W = _workload(n_il, 5, 260)
    g = dataclasses.replace(geometry_for(W), precision=precision, compensated=compensated)
    with Migrator(0) as m:
        _context(m, W, g)
        ref = m.forward()
        v = m.variant()
        assert v == (NARROW if narrow else WIDE)
        m.set_variant(v)
        assert np.array_equal(m.forward(), ref)
        m.set_variant(NARROW)
        img = m.forward()
        m.set_variant(13)
        assert np.array_equal(m.forward(), img)
        assert m.variant() in (NARROW, 13)


@pytest.mark.parametrize("precision", ["f32", "f16"])
def test_shards_are_the_whole_image(precision):
    """A rank's slab has few tiles of its own and takes the whole problem's: its rows are the whole
    image's bit for bit."""
    W = _workload(75, 5, 260)
    g = dataclasses.replace(geometry_for(W), precision=precision)
    with Migrator(0) as m:
        _context(m, W, g)
        whole = m.forward()
        assert m.variant() == WIDE
    for world in (2, 5):
        rows = [migrate_shard(g, W.data, W.vrms_cube(), r, world)[1] for r in range(world)]
        assert np.array_equal(np.concatenate(rows), whole)


@pytest.mark.parametrize("precision,compensated", [("f32", False), ("bf16", True)])
def test_batch_of_wide_and_narrow_problems(precision, compensated):
    """Every problem of a batch takes the tiles that it takes by itself, whatever its company, in
    every mode and order: the images are equal bit for bit."""
    probs, singles = [], []
    for k, (n_il, n_xl, n_t) in enumerate([(75, 5, 260), (20, 9, 300), (9, 3, 257),
                                           (40, 30, 270), (16, 7, 130)]):
        W = _workload(n_il, n_xl, n_t, pad_xl=k % 2, seed=30 + k)
        g = dataclasses.replace(geometry_for(W), precision=precision, compensated=compensated)
        with Migrator(0) as m:
            _context(m, W, g)
            singles.append(m.forward())
            assert m.variant() == (WIDE if k in (0, 3) else NARROW)
        probs.append(Problem(g, W.data, W.vrms_cube()))
    with Migrator(0) as m, Batch(m, probs) as b:
        for mode in (Batch.PERSISTENT, Batch.PER_PROBLEM, Batch.ONE_GRID):
            for order in (Batch.DEPTH_FIRST, Batch.PROBLEM_ORDER):
                b.set_mode(mode)
                b.set_order(order)
                for rep in range(2):  # capture, then replay of the graph
                    b.run()
                    for i, img in enumerate(singles):
                        assert np.array_equal(b.image(i), img), (mode, order, rep, i)
        b.set_variant(NARROW)  # one launch again
        b.run()
        assert np.array_equal(b.image(1), singles[1])
        assert b.variant() == NARROW
