"""The on-chip PSOR solve at the edges of its forms: one warp, one block,
components split over the team, more contacts than fit on chip.

Bar: impulses and states within 1e-10 of the array's largest magnitude of the
FP64 oracle, which solves the same coloured order sequentially (the device
makes the same sweeps in the same order); pair lists and colours identical.
"""
import numpy as np
import pytest

from helpers import make_pair, packed_scene, rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-10


# contacts per case (found by the oracle): 1-16 solve in one warp, up to 256
# in one block, up to 1024 split over the team, more on the team path
@pytest.mark.parametrize("n,d,phi,squeeze,lo,hi", [
    (300, 0.1, 0.05, 0.96, 1, 16),
    (1500, 0.1, 0.10, 0.95, 17, 256),
    (3000, 0.1, 0.10, 0.85, 257, 1024),
    (4000, 0.1, 0.12, 0.7, 1025, 100000),
])
@pytest.mark.parametrize("team", [1, 5])
def test_solve_forms_match_oracle(n, d, phi, squeeze, lo, hi, team):
    sc = packed_scene(n, d=d, phi=phi, seed=41, squeeze=squeeze)
    g, o = make_pair(sc, model="nsc", dt=5e-4, nsc_mu=0.4, nsc_velocity_iters=60, nsc_tol=1e-6, team_blocks=team)
    for k in range(2):
        g.step(1)
        o.step(1)
        pg, lg, cg = g.impulses()
        po, lo_, co = o.impulses()
        assert k > 0 or lo <= len(po) <= hi
        np.testing.assert_array_equal(pg, po)
        np.testing.assert_array_equal(cg, co)
        assert rel_err(lg, lo_) <= TOL
    sg, so = g.get_state(), o.get_state()
    for k in "xqvw":
        assert rel_err(sg[k], so[k]) <= TOL


def test_split_solve_to_the_sweep_limit_equals_one_block():
    # a tolerance that only a sweep without any change reaches: the chunks of
    # the split solve run full, the last one cut short by the limit
    # (8 + 32 + 32 + 3 sweeps)
    sc = packed_scene(3000, d=0.1, phi=0.10, seed=42, squeeze=0.85)
    out = []
    for team in (1, 7):
        g, _ = make_pair(sc, model="nsc", dt=5e-4, nsc_mu=0.6, nsc_velocity_iters=75, nsc_tol=1e-30, team_blocks=team)
        st = g.step(3)
        out.append((g.get_state(), g.impulses(), st))
    assert out[0][2]["psor_sweeps"] == out[1][2]["psor_sweeps"] > 3 * 40
    for k in "xqvw":
        np.testing.assert_array_equal(out[0][0][k], out[1][0][k])
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)
