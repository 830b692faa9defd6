"""The tree's point sort on both sides of its edges: one tile (4096 words, or 8192
above 16 x 512 words per SM), a look-back group of 32 tiles, and the sort of whole
keys with their indices (4096 pairs to a tile) that trees deeper than 16 levels take."""
import numpy as np
import pytest

from conftest import has_gpu
from test_gpu_sort import check

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]


def around(*edges):
    return [e + d for e in edges for d in (-1, 0, 1)]


@pytest.mark.parametrize("n", around(4096, 3 * 4096, 32 * 4096, 64 * 4096))
def test_small_tiles(n):
    rng = np.random.default_rng(n)
    check(rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), 40)


@pytest.mark.parametrize("edge", ["first", "tile", "group"])
@pytest.mark.parametrize("d", [-1, 0, 1])
def test_large_tiles(edge, d):
    import torch
    first = 16 * 512 * torch.cuda.get_device_properties(0).multi_processor_count  # the last with 4096-word tiles
    n = {"first": first, "tile": (first // 8192 + 2) * 8192, "group": (first // 262144 + 1) * 262144}[edge] + d
    rng = np.random.default_rng(n)
    check(rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), 40)


@pytest.mark.parametrize("n", around(4096, 32 * 4096))
def test_whole_keys(n):
    """100 points in a cell of level 21, at the corner where coordinates are exact"""
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    x[-100:], y[-100:] = -1 + 2.0 ** -21 * rng.uniform(0, 1, 100), -1 + 2.0 ** -21 * rng.uniform(0, 1, 100)
    check(x, y, 40)
