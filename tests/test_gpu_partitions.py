"""Binning into partitions: one and several rounds of triangles per block, up to the partitions that
fit a block's counters and beyond, boxes on the partitions' faces, vertices outside the grid."""
import numpy as np
import pytest

import pyoracle
from ooc_svo_builder_gb300 import make_params, octree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,N,limit", [(700_001, 128, 1), (1_300_000, 128, 1), (3001, 1024, 1), (257, 512, 1),
                                           (2000, 2048, 1)])
def test_binning(builder, count, N, limit):
    rng = np.random.default_rng(count)
    v = np.repeat(rng.random((count, 1, 3), dtype=np.float32), 3, axis=1)
    big = rng.integers(0, count, 200)
    v[big, 1:] += rng.uniform(-0.02, 0.02, (200, 2, 3)).astype(np.float32)
    face = rng.integers(0, count, 300)
    v[face] = np.round(v[face] * 8) / 8  # on the slabs' bounds
    v[1::997, 1, 2] = 1.5  # outside
    t = v.reshape(-1, 9)
    got = builder.build(t, make_params(N, limit, geometry_only=True))
    nodes, data, info = pyoracle.build(t, N, limit)
    assert got.info["n_partitions"] == info["n_partitions"]
    assert not octree.diff(got.tree, octree.Octree(N, nodes, data))
