"""The benchmark's split of a workload's triangles into those of the one-thread pass and those of the line
walk: boxes of at most small_vol voxels with at most one extent above two."""
import numpy as np
import pytest

import bench


def tri_of(ext, grid):
    lo = np.float32(5.5) / grid
    hi = (np.float32(4.5) + np.asarray(ext, np.float32)) / grid
    return np.concatenate([[lo] * 3, hi, hi]).astype(np.float32)


@pytest.mark.parametrize("ext,small_vol,small", [((1, 1, 1), 1, True), ((2, 2, 4), 16, True), ((4, 2, 2), 16, True),
                                                 ((2, 2, 5), 16, False), ((1, 3, 3), 16, False), ((1, 16, 1), 16, True),
                                                 ((1, 17, 1), 16, False), ((2, 1, 32), 64, True), ((3, 3, 3), 64, False)])
def test_split(ext, small_vol, small):
    t = tri_of(ext, 64)[None]
    assert bench.split_triangles(t, 64, small_vol) == ((int(np.prod(ext)), 0) if small else (0, 1))
