"""Failed calls of the persistent Verlet step, without a GPU fault: a barrier
that waits in vain for a block (the rg_config test hook test_absent_blocks,
the ordinary bounded wait with a short limit), and a state that is not finite
in one member of a batch while another outgrows its buffers.
"""
import numpy as np
import pytest

import rodgpu
from helpers import make_pair, packed_scene, rel_err

pytestmark = pytest.mark.gpu

RG_ERR_NONFINITE, RG_ERR_TIMEOUT = 4, 7

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


def _closing_rods(n, seed):
    """Rods on their way to one point: few contacts at first, nearly every
    pair within 40 steps of 1e-3 (soft springs that hardly slow them)."""
    r = np.random.default_rng(seed)
    q = r.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    x = r.uniform(-3.0, 3.0, (n, 3))
    z = np.zeros((n, 3))
    bodies = (np.full(n, 0.1), np.full(n, 0.5), np.ones(n), np.full((n, 3), 0.1), np.full(n, 0.2))
    cfg = rodgpu.default_config(n_bodies=n, model="hertz-mindlin", dt=1e-3, hm_youngs_modulus=1.0, pbc_enabled=0,
                                gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0)
    return cfg, bodies, (x, q, -x / 0.04, z)


def test_batch_error_leaves_the_other_members_sound():
    # Member 0's velocities are not finite after its first step; members 1 and
    # 2 outgrow their lists (and member 1 its 4096 contacts) some steps later
    # in the same launch; member 3 steps on.
    cfg0, bodies, s0 = _closing_rods(30, 5)
    cfg0.gravity[0] = np.nan
    cfg0.pbc_enabled, cfg0.near_skin_pct = 1, -1
    for k in range(3):  # every pair listed for good: no grid of positions that are not finite
        cfg0.pbc_min[k], cfg0.pbc_max[k] = -1.0, 1.0
    cfg1, bodies1, s1 = _closing_rods(150, 6)
    cfg2, bodies2, s2 = _closing_rods(40, 7)
    cfg3, bodies3, s3 = _closing_rods(12, 8)
    bt = rodgpu.Batch([cfg0, cfg1, cfg2, cfg3])
    for k, (bo, st) in enumerate(((bodies, s0), (bodies1, s1), (bodies2, s2), (bodies3, s3))):
        bt.set_bodies(k, *bo)
        bt.set_state(k, *st)
    before = [bt.get_state(k) for k in range(4)]
    with pytest.raises(rodgpu.RgError) as ei:
        bt.step(40)
    assert ei.value.code == RG_ERR_NONFINITE and "member 0" in str(ei.value)
    for k in (0, 1, 2):
        now = bt.get_state(k)
        for key in now:
            np.testing.assert_array_equal(now[key], before[k][key])
    for k, cfg, bo, st, done in ((1, cfg1, bodies1, s1, 0), (2, cfg2, bodies2, s2, 0), (3, cfg3, bodies3, s3, 40)):
        m = bt.member(k)
        a = rodgpu.System(cfg)
        a.set_bodies(*bo)
        a.set_state(*st)
        if done:
            a.step(done)
        assert m.step(40)["contacts"] == a.step(40)["contacts"]
        x, y = m.get_state(), a.get_state()
        for key in x:
            np.testing.assert_array_equal(x[key], y[key])
        for h, i in zip(m.history(), a.history()):
            np.testing.assert_array_equal(h, i)
        if k == 1:
            assert len(m.history()[0]) > 4096
    bt.close()
