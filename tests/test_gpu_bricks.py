"""The brick layout against the oracle where its sizes change: stripes of fewer levels than a brick
(gridsize up to 16), of one brick, of a few; bricks that are full (many windows of records per step)
and bricks with a single voxel in a corner."""
import numpy as np
import pytest

import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri

pytestmark = pytest.mark.gpu


def corner_tris(N, payload):
    """A triangle inside one voxel for voxels at the ends of blocks, units, bricks and the grid."""
    at = sorted({k % N for k in (0, 1, 3, 4, 7, 8, 15, 16, 31, 32, N - 1)})
    cells = np.array([(x, y, z) for x in at for y in at for z in at if (x + 2 * y + 3 * z) % 5 == 0], np.float64)
    v = [((cells + d) / N).astype(np.float32) for d in ((0.3, 0.3, 0.3), (0.6, 0.3, 0.4), (0.3, 0.6, 0.6))]
    col = np.random.default_rng(N).random((3, len(cells), 3), dtype=np.float32)
    return tri.pack(*v, colors=list(col) if payload else None)


@pytest.mark.parametrize("payload,levels", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("N", [1, 2, 4, 8, 16, 32, 64, 512])
def test_bricks(builder, N, payload, levels):
    meshes = [corner_tris(N, payload)]
    if N <= 64:  # nearly every voxel set
        meshes.append(tri.random_tris(400 + 40 * N, N, payload, max_edge=0.8))
    for t in meshes:
        got = builder.build(t, make_params(N, 2048, geometry_only=not payload, levels=levels))
        nodes, data, info = pyoracle.build(t, N, 2048, levels=levels)
        d = octree.diff(got.tree, octree.Octree(N, nodes, data))
        assert not d, "\n".join(d)
        assert got.info["n_filled"] == info["n_filled"]


@pytest.mark.parametrize("payload,levels", [(False, False), (True, False), (True, True)])
def test_sparse_bricks(builder, payload, levels):
    """Scattered points: a warp takes several groups of 32 bricks, each from many words, ending inside parents."""
    at = np.random.default_rng(3).random((600000, 3), dtype=np.float32)
    t = tri.pack(at, at, at, colors=[at, at, at] if payload else None)
    got = builder.build(t, make_params(2048, 2048, geometry_only=not payload, levels=levels))
    want = octree.Octree(2048, *pyoracle.build(t, 2048, 2048, levels=levels)[:2])
    assert not octree.diff(got.tree, want)
