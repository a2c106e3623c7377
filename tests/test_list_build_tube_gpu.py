"""List builds where a rod's cell is crowded and its neighbourhood is not: rods in
a narrow tube have neighbours along one axis only, so a thread per rod has few
candidates and the build by cell costs its barriers for nothing.
"""
import numpy as np
import pytest

import rodgpu
from helpers import tube_config, tube_scene

pytestmark = pytest.mark.gpu


def test_a_tube_is_built_as_fast_as_a_box_of_the_same_rods():
    # 60 rods on one block, by the step's phase timers: 26 us a build by rod,
    # 130 by cell; a uniform box of one rod a cell takes 60 (27 cells a rod)
    def build_ms(tube):
        sc = tube_scene(60)
        kw = dict(model="nsc", team_blocks=1, nsc_velocity_iters=2, nsc_position_psor_iters=2, dt=1e-6)
        r = np.random.default_rng(1)
        if not tube:
            side = 1.2 * 60 ** (1.0 / 3.0)
            sc["box_min"], sc["box_max"], sc["tube"] = (0.0,) * 3, (side,) * 3, 10.0
        s = rodgpu.System(tube_config(sc, **kw))
        s.set_bodies(sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
        s.set_profiling(True)
        z, t = np.zeros((60, 3)), []
        for k in range(6):  # other places each time: lists are built again
            x = tube_scene(60, seed=2 + k)["x"] if tube else r.uniform(0.0, side, (60, 3))
            s.set_state(x, sc["q"], z, z)
            before = s.phase_times()["list_rebuild"]
            n = s.step(1)["list_rebuilds"]
            assert n >= 1
            t.append((s.phase_times()["list_rebuild"] - before) / n)
        return float(np.median(t[1:]))

    assert build_ms(True) < 1.5 * build_ms(False)
