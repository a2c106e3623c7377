"""State upload and download on both sides of the size from which the arrays
are turned over on the device (4096 rods): what goes in comes back bit for
bit, and a refused upload changes nothing."""
import numpy as np
import pytest

import rodgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 70001])
def test_state_round_trip_and_refusal(n):
    rng = np.random.default_rng(n)
    s = rodgpu.System(rodgpu.default_config(n_bodies=n, model="nsc", pbc_enabled=0))
    one = np.ones(n)
    s.set_bodies(0.05 * one, 0.5 * one, one, np.ones((n, 3)), 0.2 * one)
    up = {"x": rng.normal(size=(n, 3)) * 100.0, "q": rng.normal(size=(n, 4)), "v": rng.normal(size=(n, 3)),
          "w": rng.normal(size=(n, 3))}
    s.set_state(**up)
    got = s.get_state()
    for k in up:
        np.testing.assert_array_equal(got[k], up[k])
    assert not got["f"].any() and not got["tau"].any()
    for k, where in (("x", 0), ("q", n - 1), ("w", n // 2)):
        bad = {a: b.copy() for a, b in up.items()}
        bad[k] += 1.0
        bad[k][where, -1] = np.inf if k == "q" else np.nan
        with pytest.raises(rodgpu.RgError) as e:
            s.set_state(**bad)
        assert e.value.code == 4
        after = s.get_state()
        for a in up:
            np.testing.assert_array_equal(after[a], up[a])
    # forces given: the host path at every size
    f, tau = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    s.set_state(**up, f=f, tau=tau)
    got = s.get_state()
    np.testing.assert_array_equal(got["f"], f)
    np.testing.assert_array_equal(got["tau"], tau)
    s.set_state(**up)
    assert not s.get_state()["f"].any()
