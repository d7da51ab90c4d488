"""The mixed corrector's mean |v|^2 (it normalises eps_v, which decides a rerun)."""
import numpy as np
import pytest

from test_gpu_step import make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [8, 50])
@pytest.mark.parametrize("speed", [1e-3, 1e18])
def test_eps_v_whatever_the_particles_per_block(cells, speed):
    """eps_v against its definition in FP64, with 2,048 and 500,000 particles, two of the latter
    or more to a thread: at speed 1e18 a block's |v|^2 sum is beyond FP32's range.  |v|^2 and
    |dv|^2 of a particle are FP32 (at most 8 roundings of 2^-24 each, halved by the root)."""
    from shamrock_gb300 import _lib, setups

    s = setups.sedov_taylor(cells, jitter=0.05, seed=1)
    n = len(s["u"])
    s["u"] = np.full(n, 1e24 if speed > 1 else 1e-6)
    s["vel"] = np.tile([speed, 0.0, 0.0], (n, 1))
    model, _ = make_pair(s, precision="mixed")
    dt = 1e-2 / speed if speed > 1 else 1e-4
    model.set_next_dt(dt)
    log = model.evolve_once(tier=_lib.GBSPH_MIXED)
    assert log["corrector_iters"] == 1
    d = model.collect_data()
    # the accelerations before the step are zero
    dv = 0.5 * dt * np.sqrt((d["axyz"] ** 2).sum(1).max())
    want = dv / np.sqrt((d["vxyz"] ** 2).sum(1).mean())
    assert want > 0
    assert abs(log["eps_v"] - want) <= 8 * 2.0**-24 * want
