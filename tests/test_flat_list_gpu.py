"""A flat pair list that does not fit (more near pairs than its first buffer
holds) grows alone, without the neighbour lists of every rod.
"""
import numpy as np
import pytest
import torch

import rodgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near_skin_pct", [100, -1])
def test_flat_list_grows_alone(near_skin_pct):
    # 100000 rods of 128 list slots: near lists as wide as the lists hold some
    # 20 pairs a rod, the flat list starts at 16.  The lists and near lists
    # would double by 100 MB; the flat list needs 40.
    n, side = 100000, 16.2
    r = np.random.default_rng(1)
    q = r.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    x, v = r.uniform(-0.5 * side, 0.5 * side, (n, 3)), r.normal(0.0, 0.1, (n, 3))
    out = []
    for profiling in (False, True):  # the multi-kernel form has no flat list to fill
        s = rodgpu.System(rodgpu.default_config(n_bodies=n, model="hertz-mindlin", dt=1e-5, hm_youngs_modulus=1.0,
                                                gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0, skin=0.3,
                                                near_skin_pct=near_skin_pct, max_neighbors=128, pbc_enabled=1,
                                                pbc_min=(-0.5 * side,) * 3, pbc_max=(0.5 * side,) * 3))
        s.set_bodies(np.full(n, 0.05), np.full(n, 0.5), np.ones(n), np.full((n, 3), 0.1), np.full(n, 0.2))
        s.set_state(x, q, v, np.zeros((n, 3)))
        s.set_profiling(profiling)
        s.step(0)  # the snapshot's buffers
        s.get_state()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        st = s.step(2)
        torch.cuda.synchronize()
        grown = free - torch.cuda.mem_get_info()[0]
        if not profiling:
            assert 30e6 < grown < 70e6, grown
        out.append((st["contacts"], s.get_state()))
        s.close()
    assert out[0][0] == out[1][0] > 1000
    for k in out[0][1]:
        np.testing.assert_array_equal(out[0][1][k], out[1][1][k])
