"""Small triangles in boxes of one or two voxels by one to 33 along each axis, across leaf words,
bricks and partitions, degenerate ones among them; the one-per-thread pass at its thresholds."""
import numpy as np
import pytest

import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri

pytestmark = pytest.mark.gpu


def boxes(axis, longest, count, grid, seed):
    rng = np.random.default_rng(seed)
    size = rng.uniform(0.0, 1.0, (count, 3))
    size[:, axis] = rng.uniform(0.0, longest - 1.0, count)
    lo = rng.uniform(0.0, grid - 1.0 - size)
    lo[::5] = np.floor(lo[::5])  # corners on voxel faces
    v = lo[:, None] + rng.uniform(0.0, 1.0, (count, 3, 3)) * size[:, None]
    v[::7, 2] = v[::7, 1]        # a line
    v[1::49, 1:] = v[1::49, :1]  # a point
    return (v / grid).astype(np.float32)


@pytest.mark.parametrize("payload", [False, True])
@pytest.mark.parametrize("small_vol", [1, 2, 16, 64])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_orientations(builder, axis, small_vol, payload):
    grid, limit = 128, 1  # eight partitions
    v = np.concatenate([boxes(axis, n, 600, grid, 100 * axis + n) for n in (1, 2, 5, 17, 33)])
    t = v.reshape(-1, 9)
    if payload:
        t = tri.pack(*v.transpose(1, 0, 2), colors=list(np.random.default_rng(9).random(v.shape, dtype=np.float32)
                                                        .transpose(1, 0, 2)))
    old, tuned = builder.tuning(), builder.tuning()
    tuned.small_vol = small_vol
    try:
        builder.set_tuning(tuned)
        got = builder.build(t, make_params(grid, limit, geometry_only=not payload))
    finally:
        builder.set_tuning(old)
    want = octree.Octree(grid, *pyoracle.build(t, grid, limit)[:2])
    assert not octree.diff(got.tree, want)
