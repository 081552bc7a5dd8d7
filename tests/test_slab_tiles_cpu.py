"""A slab's geometry carries the tiles of the whole problem (they set the order of an output
sample's sum), whatever the slab's own size; a slab of a slab keeps them."""
import dataclasses

import numpy as np
import pytest

from poststackmig3d_b200.migration import plan_geometry, slab_geometry, split_slabs

AUTO, WIDE, NARROW = 0, 1, 2


@pytest.mark.parametrize("n_il,n_xl,n_t,pad_il,tiles", [
    (148, 14, 200, 0, WIDE), (147, 14, 200, 0, NARROW),   # 148 wide tiles fill the GPU
    (147, 14, 200, 9, NARROW),                            # repeated rows do not count
    (147, 15, 200, 0, WIDE), (74, 14, 257, 0, WIDE),
    (400, 4, 900, 0, NARROW), (400, 5, 900, 0, WIDE)])    # up to 4 crosslines: narrow
def test_slab_takes_the_whole_problems_tiles(n_il, n_xl, n_t, pad_il, tiles):
    g = plan_geometry(n_il, n_xl, n_t, 0.004, 25.0, 25.0, 30.0, 2000.0, pad_il, 0)
    assert g.tiles == AUTO and g.to_c().tiles == AUTO
    for parts in (1, 2, 7):
        for slab in split_slabs(g, parts):
            loc = slab_geometry(g, slab)
            assert loc.tiles == tiles and loc.to_c().tiles == tiles
            for inner in split_slabs(loc, 2):
                if inner[1] > inner[0]:
                    assert slab_geometry(loc, inner).tiles == tiles


def test_out_centers_that_repeat_count_once():
    g = plan_geometry(200, 14, 100, 0.004, 25.0, 25.0, 30.0, 2000.0)
    g = dataclasses.replace(g, out_center=np.repeat(np.arange(100), 2).astype(np.int32))
    assert slab_geometry(g, split_slabs(g, 3)[0]).tiles == NARROW
