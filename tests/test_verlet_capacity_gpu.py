"""Full buffers inside a call of the persistent Verlet step, against the
multi-kernel form bit for bit: more contacts than the contact buffer (4096 at
least), more history entries than the table (8192), and a table that fills up
with ended contacts, which the kernel removes without growing it.
"""
import numpy as np
import pytest

import rodgpu

pytestmark = pytest.mark.gpu

MODELS = {
    "hm": dict(model="hertz-mindlin", hm_youngs_modulus=1e-3),
    "cundall": dict(model="harmonic", soft_k_scaler=1e-3, soft_damping=1e-3, soft_friction_mode="cundall"),
}


def _rods(n, side, seed):
    r = np.random.default_rng(seed)
    q = r.normal(size=(n, 4))
    return r, r.uniform(-0.5 * side, 0.5 * side, (n, 3)), q / np.linalg.norm(q, axis=1, keepdims=True)


def _pair(n, d, x, q, v, **kw):
    """The same system in the persistent and in the multi-kernel form."""
    out = []
    for profiling in (False, True):
        s = rodgpu.System(rodgpu.default_config(n_bodies=n, dt=1e-3, gravity=(0.0, 0.0, 0.0), lin_damp=0.0,
                                                ang_damp=0.0, **kw))
        s.set_bodies(np.full(n, 0.5 * d), np.full(n, 0.5), np.ones(n), np.full((n, 3), 0.1), np.full(n, 0.2))
        s.set_state(x, q, v, np.zeros((n, 3)))
        s.set_profiling(profiling)
        out.append(s)
    return out


def _same(a, b, steps):
    st, su = a.step(steps), b.step(steps)
    for k in ("contacts", "contact_steps", "history_size", "potential_energy"):
        assert st[k] == su[k], k
    sa, sb = a.get_state(), b.get_state()
    for k in sa:
        np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    for x, y in zip(a.history(), b.history()):
        np.testing.assert_array_equal(x, y)
    return st


@pytest.mark.parametrize("model", MODELS)
def test_contacts_outgrow_their_buffer(model):
    # 160 rods on their way to one point, where nearly all of the 12720 pairs
    # touch; the first call leaves a history behind
    r, x, q = _rods(160, 4.0, 1)
    a, b = _pair(160, 0.2, x, q, -x / 0.04, pbc_enabled=0, **MODELS[model])
    assert 0 < _same(a, b, 8)["history_size"] < 4096
    assert _same(a, b, 30)["contacts"] > 4096
    _same(a, b, 5)


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("speed,steps", [
    (200.0, 10),  # a diameter a step: all pairs are new ones
    (20.0, 60),   # a tenth of them: ended contacts fill the table
])
def test_history_fills_up(model, speed, steps):
    r, x, q = _rods(560, 3.0, 2)
    box = dict(pbc_enabled=1, pbc_min=(-1.5,) * 3, pbc_max=(1.5,) * 3)
    a, b = _pair(560, 0.2, x, q, r.normal(0.0, speed, (560, 3)), **box, **MODELS[model])
    assert 2000 < _same(a, b, steps)["contacts"] < 4096
    _same(a, b, 3)
