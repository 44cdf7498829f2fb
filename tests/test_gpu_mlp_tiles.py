"""Gradient kernel of the learned warm start at the edges of its 128-sample tiles: one
sample, one short of and one past a tile, and more tiles than the GPU has SMs."""
import os
import sys

import numpy as np
import pytest

from jitterphysics2_gb300 import learned
from jitterphysics2_gb300.world import World

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))
import mlp_ref as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 160 * 128 + 5])
def test_gradients_at_tile_edges(n):
    rng = np.random.default_rng(n)
    X = rng.normal(0, 2, (max(n, 64), M.IN)).astype(np.float32)
    T = rng.normal(0, 3, (max(n, 64), M.OUT)).astype(np.float32)
    p = learned.init_params(X, T, seed=3)
    w = World(max_bodies=16)
    w.mlp_load(p)
    g, _ = w.mlp_gradients(X[:n], T[:n])
    _, _, og = M.forward_backward(p.astype(np.float64), X[:n], T[:n])
    o = 0
    for name, shp in M.SIZES[:6]:
        k = int(np.prod(shp))
        a, b = g[o:o + k], og[o:o + k]
        # a BF16 operand on the other side of a rounding boundary differs by 2^-8 of itself,
        # in each of the three layers; a row or column in the wrong place is an error of 1
        assert np.linalg.norm(a - b) <= 3 * 2.0 ** -8 * np.linalg.norm(b) + 1e-12, name
        o += k
