"""The size of a batch's node tiles (the blocks of its closing launch and, in
the FP64 form, of every launch) changes no bit: 32, 64 and 256 nodes, and
CFD_BATCH_FACE_TILES (128 by another name), against 128, on lattices whose
last tiles are ragged."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_node_tiles_of_every_size(ctx, precision):
    from cfd_gb300 import abi, cases, runtime
    cs = [cases.taylor_green(shape=s) for s in ((11, 9, 7), (16, 8, 8), (5, 4, 3))]
    out = {}
    for tile in (128, 32, 64, 256) + ((abi.BATCH_FACE_TILES,) if precision else ()):
        b = runtime.Batch(ctx, precision)
        slots = [b.add(c) for c in cs]
        b.set_tiling(tile)
        b.step(3)
        assert b.info().tile_nodes == (128 if tile == abi.BATCH_FACE_TILES else tile)
        out[tile] = [b.get_flow(s) for s in slots]
        b.close()
    for tile, flows in out.items():
        for f, want in zip(flows, out[128]):
            assert np.array_equal(f, want), f"tiles of {tile}"
