"""The FP64 derivatives' v_sig maximum: pairs of one row whose |v.r_hat| are equal, nearly
equal, rising or falling, which take the candidates' pruning or, beyond eight a lane, the
whole row's exact evaluation."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sphere(m):
    k = np.arange(m) + 0.5
    z, phi = 1 - 2 * k / m, np.pi * (1 + 5**0.5) * k
    s = np.sqrt(1 - z * z)
    return np.stack([s * np.cos(phi), s * np.sin(phi), z], 1)


def _speeds(kind, m, rng):
    if kind == "equal":
        return np.ones(m)
    if kind == "near":
        return 1.0 + 1e-9 * rng.random(m)
    if kind == "rising":
        return np.linspace(0.5, 1.5, m)
    if kind == "rising a little":
        return 1.0 + 2e-7 * np.arange(m)
    if kind == "falling":
        return np.linspace(1.5, 0.5, m)
    k = 0.5 + rng.random(m)  # "groups": the largest value four times a lane
    k[rng.choice(m, min(m, 16), replace=False)] = 1.6
    return k


@pytest.mark.parametrize("kind", ["equal", "near", "rising", "rising a little", "falling", "groups"])
@pytest.mark.parametrize("m", [8, 33, 64, 300])
def test_vsig_of_near_equal_pairs(gctx, kind, m):
    """A particle with m neighbours on a sphere about it, all pairs listed for all rows."""
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(m)
    r_hat = _sphere(m)
    n = m + 1
    pos = np.concatenate([np.zeros((1, 3)), 0.7 * r_hat])
    v = np.concatenate([np.zeros((1, 3)), -_speeds(kind, m, rng)[:, None] * r_hat])
    h = np.full(n, 0.5)
    f = dict(om=1 + 0.01 * rng.random(n), u=rng.random(n), P=rng.random(n), cs=0.1 * rng.random(n))
    csr = dict(cnt=np.full(n, n), scanned=np.arange(n) * n, entries=np.tile(np.arange(n), n))
    a, du, vs = M.derivs_constAV(gctx, M.csr_to_cuda(csr), pos, v, h, f["om"], f["u"], f["P"], f["cs"],
                                 0.1, 1.0, 1.0, 2.0)
    oa, odu = O.derivs_constAV(csr, pos, v, h, f["om"], f["u"], f["P"], f["cs"], 0.1, 1.0, 1.0, 2.0)
    ovs = O.vsig(csr, pos, v, h, f["cs"])
    assert np.array_equal(vs.cpu().numpy(), ovs)
    assert np.array_equal(a.T.cpu().numpy(), oa) and np.array_equal(du.cpu().numpy(), odu)
    assert ovs[0] > 1.0
