"""A large rod under many small ones (one body with hundreds of contacts) in the
persistent Verlet step: the sums keep the contact order, so the states are the
multi-kernel form's bit for bit, and the large rod's place among the bodies
(first or second body of its contacts) does not decide what a step costs.
"""
import time

import numpy as np
import pytest

import rodgpu

pytestmark = pytest.mark.gpu

MODELS = {
    "hm": dict(model="hertz-mindlin", hm_youngs_modulus=1e3, hm_restitution=0.5),
    "cundall": dict(model="harmonic", soft_damping=0.3, soft_friction_mode="cundall"),
}


def _hub(touching, place, static=False, **kw):
    """One rod of radius 0.3 with `touching` rods of radius 0.025 lying along
    it, and as many again out of reach; the large one first or last."""
    r = np.random.default_rng(touching)
    n = 2 * touching
    a, y = r.uniform(0.0, 2 * np.pi, touching), r.uniform(-0.7, 0.7, touching)
    x = np.stack([0.3245 * np.cos(a), y, 0.3245 * np.sin(a)], 1)
    far = r.uniform(-1.9, 1.9, (touching, 3))
    far[:, 0] = np.where(far[:, 0] < 0, far[:, 0] - 1.5, far[:, 0] + 1.5)
    x = np.concatenate([x, far])
    rad, half = np.full(n, 0.025), np.full(n, 0.1)
    at = 0 if place == "first" else n
    x = np.insert(x, at, [0.0, 0.0, 0.0], axis=0)
    rad, half = np.insert(rad, at, 0.3), np.insert(half, at, 0.8)
    mass = np.insert(np.full(n, 0.01), at, 0.0 if static else 5.0)
    inertia = np.insert(np.full((n, 3), 1e-4), at, [1.0, 1.0, 1.0], axis=0)
    q = np.tile([1.0, 0.0, 0.0, 0.0], (n + 1, 1))
    v = r.normal(0.0, 0.05, (n + 1, 3))
    s = rodgpu.System(rodgpu.default_config(n_bodies=n + 1, dt=1e-5, gravity=(0.0, 0.0, 0.0), lin_damp=0.0,
                                            ang_damp=0.0, pbc_enabled=0, max_neighbors=2048, **kw))
    s.set_bodies(rad, half, mass, inertia, np.full(n + 1, 0.2))
    s.set_state(x, q, v, np.zeros((n + 1, 3)))
    return s


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("touching,place,static", [
    (9, "last", False), (10, "last", False),  # about the length that is sorted
    (300, "last", False), (300, "last", True), (300, "first", False),
])
def test_sums_of_a_long_list_equal_multi_kernel(model, touching, place, static):
    a, b = (_hub(touching, place, static, **MODELS[model]) for _ in range(2))
    b.set_profiling(True)
    for steps in (1, 2, 20):
        st, su = a.step(steps), b.step(steps)
        assert st["contacts"] == su["contacts"] and st["contacts"] >= 0.9 * touching
        sa, sb = a.get_state(), b.get_state()
        for k in sa:
            np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
        for x, y in zip(a.history(), b.history()):
            np.testing.assert_array_equal(x, y)


def test_a_step_costs_the_same_with_the_large_rod_last():
    # a list walk for each of its 900 contacts took 20 ms a step with the large
    # rod last, against 1 with it first
    def ms(place):
        s = _hub(900, place, **MODELS["hm"])
        s.step(2)
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            s.step(5)
            t.append(time.perf_counter() - t0)
        return float(np.median(t))

    assert ms("last") < 4.0 * ms("first")
