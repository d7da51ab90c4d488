"""Neighbour cache of pairs at the pair threshold, on both sides of the line between rows
tested in FP32 first and rows decided in FP64 alone, in leaves of few rows and of many."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1.0, 3.0, 4.9, 5.1, 5.9, 6.1, 10.9, 30.0])
@pytest.mark.parametrize("at", [0.5, 1e3])
@pytest.mark.parametrize("groups,pairs", [(60, 12), (1, 400)])
def test_pairs_at_the_threshold(gctx, width, at, groups, pairs):
    """Groups of coordinates within `width` pair radii of a point (up to twice that from the
    leaf's first row, from where the rule counts), a leaf each, every particle with a partner
    at the radius times 1 + d, |d| from 1e-8 to 3e-5."""
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(int(100 * width) + pairs)
    n, radius, htol = groups * pairs, 1e-5, 1.1
    lo, hi = (at - 1.0,) * 3, (at + 1.0,) * 3
    cells = (0.5 + rng.integers(0, 1000, (groups, 3))) / 512
    p = at - 1.0 + np.repeat(cells, pairs, 0) + width * radius * (2 * rng.random((n, 3)) - 1)
    e = rng.standard_normal((n, 3))
    e /= np.sqrt((e * e).sum(1))[:, None]
    d = rng.choice([-1, 1], n) * 10 ** rng.uniform(-8, -4.5, n)
    pos = np.concatenate([p, p + (radius * (1 + d))[:, None] * e])
    h = np.full(2 * n, radius / 2 / htol)
    oc = O.Tree(pos, lo, hi, 0, h=h, htol=htol).neigh_cache(pos, h, 2 * n, htol)
    for precision in ("mixed", "fp64"):
        M.Tree(gctx, pos, lo, hi, 0, h=h, htol=htol)
        csr = M.neighbour_cache(gctx, 2 * n, htol, precision)
        for key in ("cnt", "scanned", "entries"):
            assert np.array_equal(csr[key].cpu().numpy().view(np.uint32), oc[key]), (precision, key)
