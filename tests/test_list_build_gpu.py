"""Neighbour lists built inside the persistent kernels and by the plain
launches, at the edges of the rule that picks the form of the build: a thread
per rod (more than 2048 rods a block, fewer than 16 a cell), a block per home
cell, and the in-order lists of a box where every pair is listed.  The contact
query that follows draws on the lists as they are; its pairs are the oracle's.
"""
import numpy as np
import pytest

from helpers import make_pair, packed_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,phi,team", [
    (2, 0.2, 0.3, 0), (33, 0.2, 0.3, 1), (33, 1.0, 0.05, 2), (129, 1.0, 0.05, 5),  # every pair listed
    (2048, 0.2, 0.1, 1), (2049, 0.2, 0.1, 1), (4097, 0.2, 0.1, 2),  # by cell, by rod, by rod
    (2049, 1.0, 0.1, 1), (700, 1.0, 0.05, 3), (1300, 1.0, 0.1, 148),  # by cell: crowded, few rods a block
])
@pytest.mark.parametrize("pbc", [1, 0])
@pytest.mark.parametrize("form", ["persistent", "nsc", "plain"])
def test_pairs_equal_oracle(n, L, phi, team, pbc, form):
    sc = packed_scene(n, L=L, d=0.1, phi=phi, seed=71, squeeze=0.9)
    kw = dict(model="nsc" if form == "nsc" else "hertz-mindlin", team_blocks=team, dt=1e-6)
    if not pbc:
        kw["pbc_enabled"] = 0
    g, o = make_pair(sc, **kw)
    if form == "nsc":  # lists built by the step's team; its motion is far below the skin
        g.step(1)
        st = g.get_state()
        o.set_state(st["x"], st["q"], st["v"], st["w"])
    else:
        g.set_profiling(form == "plain")  # stage timers need plain launches
        g.compute_forces()
    got, want = g.detect(0.0), o.detect(0.0)
    np.testing.assert_array_equal(got[0], want[0])
    assert n < 100 or len(want[0])
