"""Omega is taken once per step, at the h of the last sub-cycle, however many there were."""
import numpy as np
import pytest

from test_gpu_step import make_pair

pytestmark = pytest.mark.gpu


def _omega_passes(ctx):
    return ctx.profile_read()["omega"][1]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("cells", [8, 35])
def test_one_omega_pass_per_step(precision, fused, cells):
    """A first step of several sub-cycles (h started at half its size), a step of one, and a
    step of several after it, which may have taken Omega ahead once: up to 1,024 rows an SM
    (2,048 rows) and beyond (171,500)."""
    from shamrock_gb300 import setups

    s = setups.sedov_taylor(cells, jitter=0.05, seed=3)
    h = s["h"].copy()
    s["h"] = 0.5 * h
    model, sim = make_pair(s, precision=precision)
    model.cfg.epsilon_h = 1e-6 if fused else 1e-5
    got = []
    for k in range(3):
        if k == 2:
            model.get_field_tensor("hpart").mul_(0.5)
        model._lib().profile(True)
        log = model.evolve_once()
        got.append((log["h_subcycles"], _omega_passes(model._lib())))
        model._lib().profile(False)
        if k == 0 and precision == "fp64" and fused:
            sim.evolve_once()
            a, b = model.collect_data(), sim.get()
            assert all(np.array_equal(a[q], b[q]) for q in ("hpart", "omega", "axyz"))
    assert got[0][0] > 2 and got[1][0] == 1 and got[2][0] > 2, got
    ahead = precision == "mixed" and fused and cells == 8
    assert [p for _, p in got] == [1, 1, 2 if ahead else 1], got


def test_omega_ahead_is_the_last_h():
    """Mixed steps whose Omega ran ahead and was taken again agree with the FP64 steps from the
    same states to the tier's 1e-5."""
    from shamrock_gb300 import setups

    out = []
    for precision in ("mixed", "fp64"):
        model, _ = make_pair(setups.sedov_taylor(8, jitter=0.05, seed=3), precision=precision)
        model.set_next_dt(0.0)
        model.evolve_once()
        model.get_field_tensor("hpart").mul_(0.5)
        model.set_next_dt(0.0)
        log = model.evolve_once()
        assert log["h_subcycles"] > 2
        out.append(model.collect_data())
    for k in ("hpart", "omega", "axyz", "duint"):
        assert np.abs(out[0][k] - out[1][k]).max() <= 1e-5 * np.abs(out[1][k]).max(), k
