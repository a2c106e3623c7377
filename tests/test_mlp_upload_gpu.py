"""Loading a network: the BF16 copies that inference reads are made from the
parameters of this very call, on a fresh system too (every system gives the
same bits)."""
import numpy as np
import pytest

import rodgpu

pytestmark = pytest.mark.gpu


def test_loaded_parameters_reach_inference_on_fresh_systems():
    rng = np.random.default_rng(3)
    f = rng.normal(0.0, 1.0, (500, 8)).astype(np.float32)
    out = []
    for _ in range(24):
        s = rodgpu.System(rodgpu.default_config(n_bodies=16, model="nsc"))
        p = np.random.default_rng(4).normal(0.0, 0.2, s.mlp_param_count()).astype(np.float32)
        s.mlp_set_params(p)
        out.append(s.mlp_infer(f))
        s.close()
    assert np.abs(out[0]).max() > 0
    for o in out[1:]:
        np.testing.assert_array_equal(o, out[0])
