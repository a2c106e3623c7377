"""Neighbour-list builds of teams where cells outnumber rods: the pairs are the
oracle's on both sides of the rule that picks the form of the build, and a
dilute system's build does not cost the walk over its empty cells.
"""
import numpy as np
import pytest

import rodgpu
from oracle import Oracle

pytestmark = pytest.mark.gpu

D, CUT = 0.1, 1.2  # diameter; cell side: rod, diameter and skin (rods of length 1)


def _quat(r, n):
    q = r.normal(size=(n, 4))
    return q / np.linalg.norm(q, axis=1, keepdims=True)


def _systems(x, q, kinds, **kw):
    n = len(x)
    cfg = rodgpu.default_config(n_bodies=n, dt=1e-6, gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0,
                                nsc_velocity_iters=2, nsc_position_psor_iters=2, **kw)
    z = np.zeros((n, 3))
    out = []
    for kind in kinds:
        s = kind(cfg)
        s.set_bodies(np.full(n, 0.5 * D), np.full(n, 0.5), np.ones(n), np.full((n, 3), 0.1), np.full(n, 0.2))
        s.set_state(x, q, z, z)
        out.append(s)
    return out


def _box(side):
    return dict(pbc_enabled=1, pbc_min=(-0.5 * side,) * 3, pbc_max=(0.5 * side,) * 3)


@pytest.mark.parametrize("model", ["nsc", "hertz-mindlin"])
@pytest.mark.parametrize("n,rho,team", [
    (257, 0.01, 1), (1000, 0.1, 8), (600, 1.0, 148),  # by rod: empty cells, one a cell, few rods a block
    (1000, 4.0, 8), (1000, 4.0, 31),                  # about rho (4 + 5 rho) rods a block: by rod, by cell
    (1500, 12.0, 2), (4096, 11.0, 4),                 # crowded cells: by cell, by rod
])
def test_pairs_of_boxes_of_every_density(model, n, rho, team):
    side = CUT * (n / rho) ** (1.0 / 3.0)
    r = np.random.default_rng(n)
    g, o = _systems(r.uniform(-0.5 * side, 0.5 * side, (n, 3)), _quat(r, n), (rodgpu.System, Oracle), model=model,
                    team_blocks=team, max_neighbors=256, **_box(side))
    if model == "nsc":
        g.step(1)
        st = g.get_state()
        o.set_state(st["x"], st["q"], st["v"], st["w"])
    else:
        g.compute_forces()
    np.testing.assert_array_equal(g.detect(0.0)[0], o.detect(0.0)[0])


@pytest.mark.parametrize("model", ["nsc", "hertz-mindlin"])
def test_pairs_of_a_cluster_with_strays(model):
    # an open box whose grid is stretched by single rods far away: a few
    # crowded cells (by cell), every other one empty or with a stray
    r = np.random.default_rng(3)
    x = np.concatenate([r.uniform(-1.5, 1.5, (500, 3)), r.uniform(-150.0, 150.0, (30, 3))])
    x = x[r.permutation(len(x))]
    g, o = _systems(x, _quat(r, len(x)), (rodgpu.System, Oracle), model=model, team_blocks=3, max_neighbors=512,
                    pbc_enabled=0)
    if model == "nsc":
        g.step(1)
        st = g.get_state()
        o.set_state(st["x"], st["q"], st["v"], st["w"])
    else:
        g.compute_forces()
    want = o.detect(0.0)[0]
    assert len(want) > 100
    np.testing.assert_array_equal(g.detect(0.0)[0], want)


def test_a_dilute_build_is_not_slower_than_a_crowded_one():
    # 1000 rods on 8 blocks, by the step's phase timers: 60 us in 32768 cells
    # and 150 in 64 (a walk over the empty cells one by one: 2100), so a factor
    # of three leaves room for noise on both sides.
    def build_ms(rho):
        side = CUT * (1000 / rho) ** (1.0 / 3.0)
        r = np.random.default_rng(1)
        (s,) = _systems(r.uniform(-0.5 * side, 0.5 * side, (1000, 3)), _quat(r, 1000), (rodgpu.System,), model="nsc", team_blocks=8,
                        max_neighbors=256, **_box(side))
        s.set_profiling(True)
        z, t = np.zeros((1000, 3)), []
        for _ in range(6):  # positions far from the ones before: lists are built again
            s.set_state(r.uniform(-0.5 * side, 0.5 * side, (1000, 3)), _quat(r, 1000), z, z)
            before = s.phase_times()["list_rebuild"]
            assert s.step(1)["list_rebuilds"] >= 1
            t.append(s.phase_times()["list_rebuild"] - before)
        return float(np.median(t[1:]))

    assert build_ms(0.03) < 3.0 * build_ms(8.0)
