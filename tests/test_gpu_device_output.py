"""Octrees that stay on the device: the records written on the host (levels above the stripes, the
root) at every height of a stripe, for one stripe and for several, and builds one after the other."""
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
