"""Allocation-free occupancy calls that may overlap on the GPU share one scratch array: they may lose
voxels to each other, but set none of their own wrongly and touch nothing else, and a call ordered
after them is complete."""
import numpy as np
import pytest

import ooc_svo_builder_gb300 as ooc
from ooc_svo_builder_gb300 import tri

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("counts", [(1 << 20, 1 << 20), (1 << 20, 70), (3000, 1)])
def test_overlapping_calls(counts):
    N = 128
    rng = np.random.default_rng(counts[1])
    words = N ** 3 // 32
    prm = ooc.make_params(N, 2048)
    tris, want = [], []

    def call(t, out, stream=0):
        assert ooc.voxelize_occupancy_noalloc(prm, t.data_ptr(), len(t), out.data_ptr(), words, stream) == ooc.OOC_OK

    for k, n in enumerate(counts):
        t = np.repeat(tri.random_tris(min(n, 2000), 3 + k, False, max_edge=0.06), -(-n // 2000), axis=0)[:n]
        tris.append(torch.from_numpy(np.ascontiguousarray(rng.permutation(t))).cuda())
        out = torch.empty(words, dtype=torch.int32, device="cuda")
        call(tris[k], out)
        torch.cuda.synchronize()
        want.append(out)
        assert int(out.count_nonzero())
    streams = [torch.cuda.Stream() for _ in counts]
    for _ in range(4):
        outs = [torch.empty(words, dtype=torch.int32, device="cuda") for _ in counts]
        torch.cuda.synchronize()
        for t, out, s in zip(tris, outs, streams):
            call(t, out, s.cuda_stream)
        torch.cuda.synchronize()
        for out, w in zip(outs, want):
            assert not int((out & ~w).count_nonzero())
    for t, w in zip(tris, want):
        out = torch.empty(words, dtype=torch.int32, device="cuda")
        call(t, out)
        torch.cuda.synchronize()
        assert torch.equal(out, w)
