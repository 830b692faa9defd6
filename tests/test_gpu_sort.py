"""The tree's point sort at the edges of its tiles (4096 and 8192 words), of a
look-back group (32 tiles) and of the point counts where the tile size changes: each
point must come out in the leaf whose cell holds it, and each leaf hold its count."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]


def check(x, y, cutoff):
    import pykifmm2d_b200 as P
    kern = P.LaplaceKernel()
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 8, cutoff)
    f.build_tree()
    nodes, pl = f.export_tree()
    side = 2.0 ** pl[:, 0]  # cells of [-1, 1] per side at the leaf's level
    np.testing.assert_array_equal(pl[:, 1], np.floor((x + 1) / 2 * side))
    np.testing.assert_array_equal(pl[:, 2], np.floor((y + 1) / 2 * side))
    leaves = nodes[(nodes[:, 3] == 1) & (nodes[:, 6] > 0)]
    cells, counts = np.unique(pl, axis=0, return_counts=True)  # sorted as the nodes are
    np.testing.assert_array_equal(cells, leaves[:, :3])
    np.testing.assert_array_equal(counts, leaves[:, 6])


def tile_edges():
    import torch
    wave = 512 * (torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148)
    return {"1": 1, "2": 2, "31": 31, "2047": 2047, "2048": 2048, "2049": 2049, "65536": 65536, "65537": 65537,
            "4 waves": 4 * wave, "4 waves + 1": 4 * wave + 1, "16 waves": 16 * wave, "16 waves + 1": 16 * wave + 1,
            "19 waves + 77": 19 * wave + 77}


@pytest.mark.parametrize("size", ["1", "2", "31", "2047", "2048", "2049", "65536", "65537", "4 waves", "4 waves + 1",
                                  "16 waves", "16 waves + 1", "19 waves + 77"])
def test_points_in_their_leaves(size):
    n = tile_edges()[size]
    rng = np.random.default_rng(n)
    check(rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), 40)


def test_one_digit():
    """Every key in one cell of level 8: each pass has a digit that all keys share."""
    rng = np.random.default_rng(0)
    h = 2.0 ** -7
    x, y = rng.uniform(0, h, 70_000), rng.uniform(0, h, 70_000)
    x[0], y[0], x[1], y[1] = -0.9, -0.9, 0.9, 0.9
    check(x, y, 60)
