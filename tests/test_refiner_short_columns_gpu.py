"""The weight gradient's rings where a block takes many short columns: images of few
rows and batches of many, so that every level's share of a block crosses columns of
1, 2, 3 rows or more (rows without dZ come two a column, and the warps that sum the
bias have no part in them)."""
import importlib

import numpy as np
import pytest

from test_refiner_edges_gpu import test_each_layer_at_tile_edges as each_layer

pytestmark = pytest.mark.gpu

SIZES = [(1216, 8, 8), (700, 16, 8), (460, 24, 8), (300, 48, 8)]


@pytest.mark.parametrize("n,h,w", SIZES)
def test_each_layer_of_many_short_columns(cuda, n, h, w):
    """Every layer within the bounds derived for the tile edges: a block adds at
    most one partial sum per 16 pixels here too (fewer than 200)."""
    each_layer(cuda, n, h, w)


@pytest.mark.parametrize("n,h,w", SIZES)
def test_short_columns_give_the_same_bits_every_time(cuda, n, h, w):
    rf = importlib.import_module("3deye_gb300.refiner")
    rng = np.random.default_rng(n)
    raw = rng.integers(500, 3000, (n, h, w)).astype(np.uint16)
    tgt = np.clip(raw.astype(np.int64) + rng.integers(-6, 7, raw.shape), 0, 32767).astype(np.uint16)
    R = rf.Refiner(n, h, w, seed=3)
    first = None
    for _ in range(12):
        R.loss_grad(raw, tgt)
        assert R.status() == 0
        g = R.grads().view(np.uint32).copy()
        first = g if first is None else first
        assert np.array_equal(g, first)
    R.close()
