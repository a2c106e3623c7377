"""The balanced schedule's cost model where a member's solves are split over its
team (more than 256 contacts): they count as work that more blocks shorten, not
as the floor of the plan.
"""
import pytest

import rodgpu
from helpers import packed_scene
from rodgpu import scene

pytestmark = pytest.mark.gpu


def test_a_split_solve_does_not_take_the_small_members_blocks():
    # One member of some 650 contacts, twelve of a few dozen.  Taken as serial
    # time, the large one's solves left the plan only its detection to
    # shorten: it got 136 to 146 of 148 blocks, and the others two or three
    # between them.
    scs = [packed_scene(4000, phi=0.12, seed=1)] + [packed_scene(300, phi=0.05, squeeze=0.9, seed=k)
                                                    for k in range(2, 14)]
    b = rodgpu.Batch([rodgpu.default_config(n_bodies=sc["n"], model="nsc", dt=5e-4, gravity=(0.0, 0.0, 0.0),
                                            lin_damp=0.0, ang_damp=0.0, **scene.pbc_kwargs(sc)) for sc in scs])
    for k, sc in enumerate(scs):
        b.set_bodies(k, sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
        b.set_state(k, sc["x"], sc["q"], sc["v"], sc["w"])
    start = b.get_state_all()
    for _ in range(4):
        b.set_schedule(-1)  # plans again, with the times of the calls before
        b.set_state_all(*start)
        st = b.step(6)
    assert 256 < st[0]["contacts"] <= 1024
    _, blocks = b.costs()
    assert 4 <= blocks[0] <= 100, blocks
    b.close()
