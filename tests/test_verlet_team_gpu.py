"""The persistent Verlet step (one launch per call, teams of blocks) against
the multi-kernel form of the same step, bit for bit.

The stage timers need plain launches, so a system with profiling on steps in
the multi-kernel form (which tests/test_gpu_parity.py's oracle bar covers
through the small systems of both forms).  Compared after every call: states,
forces, contacts and energy, and the tangential-history table (pairs, values
and last frames: new pairs, ended contacts within and past their retention).
"""
import numpy as np
import pytest

from helpers import packed_scene
import rodgpu
from rodgpu import scene

pytestmark = pytest.mark.gpu


def _load(sc, **kw):
    base = dict(gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0)
    base.update(scene.pbc_kwargs(sc))
    base.update(kw)
    s = rodgpu.System(rodgpu.default_config(n_bodies=sc["n"], **base))
    s.set_bodies(sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
    s.set_state(sc["x"], sc["q"], sc["v"], sc["w"])
    return s


def _same(a, b):
    sa, sb = a.get_state(), b.get_state()
    for k in ("x", "q", "v", "w", "f", "tau"):
        np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    for x, y in zip(a.history(), b.history()):
        np.testing.assert_array_equal(x, y)


HM = dict(model="hertz-mindlin", dt=1e-4, hm_youngs_modulus=1e5, hm_poisson_ratio=0.3, hm_restitution=0.5,
          hm_friction=0.5)
SOFT = dict(model="harmonic", dt=1e-4, soft_damping=0.3, soft_friction_mode="cundall")


@pytest.mark.parametrize("model", [HM, SOFT], ids=["hm", "cundall"])
@pytest.mark.parametrize("n,d,phi,squeeze,team,extra", [
    (37, 0.1, 0.02, 0.8, 0, {}),                        # every pair listed and tested, one partly filled block
    (580, 0.05, 0.08, 0.9, 0, {}),                      # every pair listed, near lists drawn from them
    (300, 0.1, 0.05, 0.9, 1, dict(pbc_enabled=0)),      # open box, one block
    (1500, 0.1, 0.10, 0.95, 3, dict(skin=0.02)),        # 500 rods a block, lists rebuilt in the call
    (1300, 0.1, 0.10, 0.95, 1, {}),                     # several rods and pairs a thread
    (1500, 0.1, 0.10, 0.95, 0, dict(near_skin_pct=-1)),  # full lists instead of near lists
    (4000, 0.1, 0.12, 0.7, 0, {}),                      # more new pairs at once than are sorted on chip
])
def test_persistent_equals_multi_kernel(model, n, d, phi, squeeze, team, extra):
    sc = packed_scene(n, d=d, phi=phi, seed=51, squeeze=squeeze, sigma_v=1.0, sigma_w=1.0)
    a = _load(sc, team_blocks=team, **model, **extra)
    b = _load(sc, **model, **extra)
    b.set_profiling(True)
    contacts = set()
    for steps in (1, 2, 25, 1, 40):
        st, su = a.step(steps), b.step(steps)
        for k in ("contacts", "contact_steps", "history_size", "potential_energy", "kinetic_energy"):
            assert st[k] == su[k], k
        contacts.add(st["contacts"])
        _same(a, b)
    assert st["contacts"] > 0 and (n < 300 or len(contacts) > 1)


@pytest.mark.parametrize("model", [HM, SOFT], ids=["hm", "cundall"])
def test_near_lists_of_an_all_pairs_box_lose_no_contact(model):
    # half the box (1.22) is just above the contact reach plus the near skin;
    # fast rods: minimum images flip while the near lists are valid
    sc = packed_scene(580, d=0.05, phi=0.08, seed=54, squeeze=0.9, sigma_v=5.0, sigma_w=5.0)
    assert 2.42 < sc["side"] < 2.5
    a, b = _load(sc, **model), _load(sc, near_skin_pct=-1, **model)
    near = 0
    for _ in range(4):
        near += a.step(80)["near_rebuilds"]
        b.step(80)
        _same(a, b)
    assert near > 1


def test_switching_between_the_forms():
    sc = packed_scene(800, d=0.1, phi=0.10, seed=52, squeeze=0.93, sigma_v=0.5)
    a, b = _load(sc, **HM), _load(sc, **HM)
    b.set_profiling(True)
    for k in range(3):
        a.step(5)
        b.step(5)
        a.set_profiling(k % 2 == 0)
        fa, fb = a.compute_forces(), b.compute_forces()
        np.testing.assert_array_equal(fa[0], fb[0])
        assert fa[2] == fb[2]
        pa, pb = a.detect(0.0), b.detect(0.0)
        for x, y in zip(pa, pb):
            np.testing.assert_array_equal(x, y)
        a.step(7)
        b.step(7)
        _same(a, b)


def test_small_contact_buffers_grow_inside_a_call():
    # 16 list slots a rod overflow at once and the call starts over
    sc = packed_scene(1000, d=0.2, phi=0.25, seed=53, squeeze=0.75, sigma_v=0.5)
    a, b = _load(sc, max_neighbors=4, **HM), _load(sc, **HM)
    b.set_profiling(True)
    a.step(10)
    b.step(10)
    _same(a, b)


def test_batch_of_more_verlet_members_than_blocks_equals_members_alone():
    # 160 members: single-block teams that run several members in turn
    scs = [packed_scene(40 + k % 7, d=0.1, phi=0.04, seed=60 + k, squeeze=0.85, sigma_v=0.5) for k in range(160)]
    kws = []
    for k, sc in enumerate(scs):
        kw = dict(gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0, **(HM if k % 2 else SOFT))
        kw.update(scene.pbc_kwargs(sc))
        kws.append(kw)
    bt = rodgpu.Batch([rodgpu.default_config(n_bodies=sc["n"], **kw) for sc, kw in zip(scs, kws)])
    for k, sc in enumerate(scs):
        bt.set_bodies(k, sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
        bt.set_state(k, sc["x"], sc["q"], sc["v"], sc["w"])
    bt.step(3)
    st = bt.step(4)
    for k in range(0, 160, 13):
        s = _load(scs[k], **(HM if k % 2 else SOFT))
        s.step(3)
        su = s.step(4)
        assert st[k]["contacts"] == su["contacts"]
        a, b = bt.get_state(k), s.get_state()
        for key in "xqvw":
            np.testing.assert_array_equal(a[key], b[key])
    bt.close()
