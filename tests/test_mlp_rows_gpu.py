"""Gradients of the training kernel at the edges of its 16-row groups and
64-row tiles, and where a block takes a second tile (more than 296 tiles),
against the CPU oracle, with the bounds of the 512-row comparison."""
import numpy as np
import pytest

import mlp_oracle as M
import rodgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 16, 63, 65, 130, 19009])
def test_gradient_at_tile_edges(n):
    s = rodgpu.System(rodgpu.default_config(n_bodies=16, model="nsc"))
    x, y = M.synthetic_records(n + 64, seed=31)
    P = M.init_params(x, y, seed=32)
    s.mlp_set_params(P)
    x, y = x[:n], y[:n]
    g, loss = s.mlp_grad(x, y)
    loss_o, g_o = M.loss_and_grad(P, x, y, emulate_bf16=True)
    assert abs(loss - loss_o) / loss_o < 1e-2
    edges = [M.OFF_W1, M.OFF_B1, M.OFF_W2, M.OFF_B2, M.OFF_W3, M.OFF_B3, M.OFF_W4, M.OFF_B4, M.OFF_IN_MEAN]
    for lo, hi in zip(edges, edges[1:]):
        a, b = g[lo:hi].astype(np.float64), g_o[lo:hi]
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 2e-2, lo
    assert np.all(g[M.OFF_IN_MEAN:] == 0)
