"""Step arguments that are refused before anything runs, leaving the state as it is."""
import numpy as np
import pytest

from test_gpu_step import make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("used", [False, True])
def test_no_h_subcycles_is_refused(precision, used):
    """h_max_subcycles 0 leaves no rows, cache or h to step with: an argument error, in a new
    context and in one that has stepped, and the next step runs as if it had not been asked."""
    import shamrock_gb300.setups as setups

    model, sim = make_pair(setups.sedov_taylor(8, jitter=0.05, seed=1), precision=precision)
    if used:
        model.evolve_once()
        sim.evolve_once()
    before, t, dt = model.collect_data(), model.get_time(), model.get_dt()
    model.cfg.h_max_subcycles_count = 0
    with pytest.raises(RuntimeError, match="h_max_subcycles"):
        model.evolve_once()
    after = model.collect_data()
    for k in before:
        assert np.array_equal(before[k], after[k], equal_nan=True), k
    assert (model.get_time(), model.get_dt()) == (t, dt)
    model.cfg.h_max_subcycles_count = 100
    model.evolve_once()
    sim.evolve_once()
    a, b = model.collect_data(), sim.get()
    if precision == "fp64":
        assert all(np.array_equal(a[k], b[k]) for k in ("xyz", "vxyz", "axyz", "hpart", "uint", "duint"))
