"""Builds of one context on several streams: its own and the caller's in turn, and a device build on
another stream straight after a build that failed with kernels queued."""
import ctypes

import pytest

import ooc_svo_builder_gb300 as ooc
import pyoracle
from ooc_svo_builder_gb300 import make_params, octree, tri

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def device_build(builder, t, N, limit, stream, **kw):
    dev = torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    info = builder.build_device(dev.data_ptr(), len(t), make_params(N, limit, geometry_only=t.shape[1] == 9, **kw), stream)
    nodes, data, _ = pyoracle.build(t, N, limit, **kw)
    got = builder.result_tree(N, info["n_nodes"], info["n_data"])
    assert not octree.diff(got, octree.Octree(N, nodes, data))


@pytest.mark.parametrize("N,limit,payload,levels", [(64, 2048, False, False), (512, 2048, True, True), (256, 1, True, False),
                                                    (256, 1, False, True)])
def test_streams_in_turn(builder, N, limit, payload, levels):
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for k, (s, count) in enumerate(zip((0, a, b, 0, b, a), (40, 6000, 1, 900, 9000, 25))):
        t = tri.random_tris(count, 70 + k, payload, max_edge=0.05)
        device_build(builder, t, N, limit, s and s.cuda_stream, levels=levels)
        assert not s or s.query()  # the call returns after the stream has drained


@pytest.mark.parametrize("refuse", [0, 3, 7])
def test_other_stream_after_a_failed_batch(builder, refuse):
    """The batch runs in several sub-batches, so the refusal of a finished mesh finds the next one's kernels queued."""
    meshes = [tri.icosphere_tris(5, seed=40 + i, payload=True) for i in range(8)]
    params = [make_params(512, 2048, geometry_only=False) for _ in meshes]
    t = tri.icosphere_tris(4, seed=60, payload=True)
    s = torch.cuda.Stream()
    buf = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    arr, keep = builder._mesh_array(meshes, params)
    fn = ctypes.cast(builder.lib.ooc_arena_alloc, ctypes.c_void_p)
    ready = ooc.READY(lambda user, mesh: 1 if mesh == refuse else 0)
    budget = builder.lib.ooc_batch_budget(builder.h)
    builder.lib.ooc_set_batch_budget(builder.h, 40 << 20)
    try:
        arena = ooc.DeviceArena(buf.data_ptr(), buf.numel(), 0)
        rc = builder.lib.ooc_build_batch_device(builder.h, arr, len(meshes), fn, ctypes.cast(ready, ctypes.c_void_p),
                                                ctypes.byref(arena), (ooc.BuildInfo * len(meshes))())
        assert rc == 5  # OOC_ERR_SINK
        device_build(builder, t, 512, 2048, s.cuda_stream)
    finally:
        builder.lib.ooc_set_batch_budget(builder.h, budget)
