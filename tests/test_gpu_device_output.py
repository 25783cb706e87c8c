"""Octrees that stay on the device: the records written on the host (levels above the stripes, the
root) at every height of a stripe, for one stripe and for several, and builds one after the other."""
import numpy as np
import pytest

import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("payload,levels", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("N,limit", [(1, 2048), (2, 2048), (4, 2048), (8, 2048), (16, 2048), (32, 2048), (64, 2048),
                                     (128, 1), (256, 1), (2048, 2048)])
def test_device_output(builder, N, limit, payload, levels):
    torch = pytest.importorskip("torch")
    for count in (300, 1, 40):
        t = tri.random_tris(count, N + count, payload, max_edge=0.3 if N < 2048 else 0.01)
        dev = torch.from_numpy(t).cuda()
        info = builder.build_device(dev.data_ptr(), count, make_params(N, limit, geometry_only=not payload, levels=levels))
        nodes, data, want = pyoracle.build(t, N, limit, levels=levels)
        got = builder.result_tree(N, info["n_nodes"], info["n_data"])
        assert not octree.diff(got, octree.Octree(N, nodes, data))
        assert info["n_filled"] == want["n_filled"] and info["n_partitions"] == want["n_partitions"]


@pytest.mark.parametrize("order", [(1_200_000, 40, 0, 500_000, 3000, 700_000), (40, 900_000, 300_000, 0, 800_000, 5),
                                   (5, 0, 7, 2_000_000)])
def test_batch_in_two_parts(builder, order):
    """Device batches of more than 64 MB of triangles run a first part while the rest is on its way:
    the part's end before and after meshes without triangles, partitioned ones, one mesh of nearly everything."""
    rng = np.random.default_rng(len(order))
    meshes, params = [], []
    for i, count in enumerate(order):
        at = np.repeat(rng.random((count, 1, 3), dtype=np.float32), 3, axis=1)
        if count and count < 10_000:
            at[:, 1:] += rng.uniform(-0.1, 0.1, (count, 2, 3)).astype(np.float32)
        meshes.append(at.reshape(-1, 9))
        params.append(make_params(128 if i % 2 else 64, 1 if i % 3 == 0 else 2048, geometry_only=True))
    assert sum(m.nbytes for m in meshes) >= 64 << 20
    for _ in range(2):
        for t, p, got in zip(meshes, params, builder.build_batch_device(meshes, params)):
            nodes, data, info = pyoracle.build(t, int(p.gridsize), int(p.memory_limit_mb))
            assert not octree.diff(got.tree, octree.Octree(int(p.gridsize), nodes, data))
            assert got.info["n_filled"] == info["n_filled"]
