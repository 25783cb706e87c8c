"""The list of large triangles at its edges: triangles of many tasks, a full list of the many-task
ones, fewer triangles than warps, and triangles just over the threshold."""
import numpy as np
import pytest

import ooc_svo_builder_gb300 as ooc
import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri
from test_zz_no_alloc import noalloc_occupancy, regular_occupancy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("payload", [False, True])
@pytest.mark.parametrize("lines_per_lane,small_vol,count,edge", [
    (1, 1, 3, 1.4), (1, 64, 200, 0.9), (2, 27, 2000, 0.1), (64, 1, 700, 0.5), (16, 64, 1, 1.4)])
def test_tasks(builder, lines_per_lane, small_vol, count, edge, payload):
    t = tri.random_tris(count, 10 * count + lines_per_lane, payload, max_edge=edge)
    old, tuned = builder.tuning(), builder.tuning()
    tuned.lines_per_lane, tuned.small_vol = lines_per_lane, small_vol
    try:
        builder.set_tuning(tuned)
        got = builder.build(t, make_params(64, 2048, geometry_only=not payload))
    finally:
        builder.set_tuning(old)
    want = octree.Octree(64, *pyoracle.build(t, 64, 2048)[:2])
    assert not octree.diff(got.tree, want)


def test_full_list_of_many_task_triangles():
    # The allocation-free pass lists 4,096 triangles of more than 512 lines; one warp walks each of the others.
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    c = rng.uniform(0.45, 0.55, size=(6000, 1, 3))
    t = (c + rng.choice([-0.4, 0.4], size=(6000, 3, 3)) * rng.uniform(0.7, 1.0, size=(6000, 3, 3))).astype(np.float32)
    t = t.reshape(6000, 9)
    assert np.array_equal(noalloc_occupancy(torch, t, 64, False), regular_occupancy(t, 64, False))
    with ooc.Builder(0) as b:  # and the regular pass against the oracle on some of them
        got = b.build(t[:64], make_params(64, 2048, geometry_only=True))
    assert not octree.diff(got.tree, octree.Octree(64, *pyoracle.build(t[:64], 64, 2048)[:2]))
