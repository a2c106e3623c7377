"""Failed calls of the persistent Verlet step, without a GPU fault: a barrier
that waits in vain for a block (the rg_config test hook test_absent_blocks,
the ordinary bounded wait with a short limit).
"""
import numpy as np
import pytest

import rodgpu
from helpers import make_pair, packed_scene, rel_err

pytestmark = pytest.mark.gpu

RG_ERR_TIMEOUT = 7

HM = dict(model="hertz-mindlin", dt=1e-4, hm_youngs_modulus=1e5)
SOFT = dict(model="harmonic", dt=1e-4, soft_damping=0.3, soft_friction_mode="cundall")


@pytest.mark.parametrize("model", [HM, SOFT], ids=["hm", "cundall"])
@pytest.mark.parametrize("team_blocks", [1, 3])
def test_barrier_timeout_leaves_the_handle_as_it_was(model, team_blocks):
    sc = packed_scene(800, d=0.1, phi=0.1, seed=41, squeeze=0.97)
    g, o = make_pair(sc, team_blocks=team_blocks, spin_limit=20000, test_absent_blocks=1, **model)
    before = g.get_state()
    for call in (g.compute_forces, lambda: g.step(3), g.compute_forces):
        with pytest.raises(rodgpu.RgError) as ei:
            call()
        assert ei.value.code == RG_ERR_TIMEOUT
        after = g.get_state()
        for k in after:
            np.testing.assert_array_equal(after[k], before[k])
        assert len(g.history()[0]) == 0
    g2, _ = make_pair(sc, team_blocks=team_blocks, **model)  # the context is usable
    g2.step(2)
    o.step(2)
    a, b = g2.get_state(), o.get_state()
    for k in ("x", "q", "v", "w"):
        assert rel_err(a[k], b[k]) < 1e-10, k
