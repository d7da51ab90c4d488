"""The mixed derivatives' four-lane exchange with every term at work: viscosity, conduction,
du/dt and v_sig, on partial fours, odd row counts and free-boundary rows."""
import numpy as np
import pytest

from test_gpu_routes import _lattice_state, _sms
from test_gpu_step import make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 7, 3), (13, 9, 7), (32, 32, _sms() // 4), (32, 32, _sms() // 4 + 1)])
def test_rows_in_motion_mixed_vs_fp64(shape):
    """One step of the FP32 tier and of FP64 from the same state with random velocities and
    energies: every field, and the next time step (v_sig, the corrector's minimum), within the
    tier's 1e-5."""
    from shamrock_gb300 import _lib

    s = _lattice_state(*shape, 0, seed=3)
    rng = np.random.default_rng(5)
    s["vel"] = rng.standard_normal(s["vel"].shape)
    s["u"] = 0.5 + rng.random(len(s["u"]))
    out, dt = [], []
    for tier in (_lib.GBSPH_MIXED, _lib.GBSPH_FP64):
        model, _ = make_pair(s, precision="mixed", periodic=False)
        model.set_next_dt(0.0)
        model.evolve_once(tier=tier)
        out.append(model.collect_data())
        dt.append(model.get_dt())
    assert np.abs(out[1]["duint"]).max() > 0 and 0 < dt[1] < np.inf
    for key in ("hpart", "omega", "axyz", "duint"):
        a, b = out[0][key], out[1][key]
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), key
    assert abs(dt[0] - dt[1]) <= 1e-5 * dt[1]
