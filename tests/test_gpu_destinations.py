"""Device destinations at 8 mod 16: node files anywhere on 8 bytes, data files where they hold only their
header records; others are refused on the host, before anything is written."""
import ctypes

import pytest

import ooc_svo_builder_gb300 as ooc
import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("N", [8, 256])
@pytest.mark.parametrize("payload,nodes_off,data_off", [(False, 8, 8), (False, 0, 8), (True, 8, 0), (True, 0, 8)])
def test_offsets(builder, N, payload, nodes_off, data_off):
    t = tri.random_tris(700, 5, payload, max_edge=0.2)
    arr, keep = builder._mesh_array([t], [make_params(N, 2048, geometry_only=not payload)])
    buf = torch.zeros(256 << 20, dtype=torch.uint8, device="cuda")
    got = {}

    def alloc(user, mesh, nb, db, stream, pn, pd):
        got.update(nb=nb, db=db, data=(nb + 511) // 256 * 256 + data_off)
        pn[0] = buf.data_ptr() + nodes_off
        pd[0] = buf.data_ptr() + got["data"]
        return 0

    rc = builder.lib.ooc_build_batch_device(builder.h, arr, 1, ctypes.cast(ooc.ALLOC(alloc), ctypes.c_void_p), None, None,
                                            (ooc.BuildInfo * 1)())
    if payload and data_off:
        assert rc == 1 and int(buf.count_nonzero()) == 0  # OOC_ERR_INVALID
        return
    assert rc == 0
    host = buf.cpu().numpy().tobytes()
    nodes, data, _ = pyoracle.build(t, N, 2048)
    tree = octree.from_bytes(N, host[nodes_off:nodes_off + got["nb"]], host[got["data"]:got["data"] + got["db"]])
    assert not octree.diff(tree, octree.Octree(N, nodes, data))
