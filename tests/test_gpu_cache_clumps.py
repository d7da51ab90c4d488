"""Neighbour caches of clumps within one Morton cell: the rows of a leaf that owns more than
128 are the work of many warps."""
import time

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _clumps(sizes, spread, rng):
    """Jittered lattices of about `sizes` particles, each within one cell of 1/1024 of the unit
    box, and two particles at its corners."""
    pos, h = [np.array([[0.0, 0, 0], [1, 1, 1]])], [np.full(2, 1e-3)]
    for k, m in enumerate(sizes):
        side = int(np.ceil(m ** (1 / 3)))
        g = np.stack(np.meshgrid(*[(np.arange(side) + 0.5) / side] * 3, indexing="ij"), -1).reshape(-1, 3)[:m]
        cell = np.floor(1024 * (0.1 + 0.8 * rng.random(3))) / 1024
        pos.append(cell + (g + 0.2 / side * (rng.random(g.shape) - 0.5)) * spread + (1 / 1024 - spread) / 2)
        h.append(np.full(m, 1.2 / side * spread))
    pos, h = np.concatenate(pos), np.concatenate(h)
    order = rng.permutation(len(h))
    return pos[order], h[order]


@pytest.mark.parametrize("sizes", [[32], [33], [64, 65], [127], [128], [129], [130] * 5, [300, 40, 700, 1, 133], [1500]])
@pytest.mark.parametrize("level", [0, 3])
@pytest.mark.parametrize("budget", [0, 1])
def test_clumped_cache_vs_oracle(sizes, level, budget):
    """Both precisions, all and some of the rows, the one-pass and (budget 1 byte) the two-pass
    build."""
    from shamrock_gb300 import _lib, modules as M

    pos, h = _clumps(sizes, 9e-4, np.random.default_rng(len(sizes) + sizes[0]))
    n, lo, hi = len(h), (0.0,) * 3, (np.nextafter(1.0, 2.0),) * 3
    ctx = _lib.Context(0)
    ctx.lib.gbsph_set_cache_budget(ctx.handle, budget)
    t = O.Tree(pos, lo, hi, level, h=h, htol=1.1)
    for rows in (n, max(1, (3 * n) // 5)):
        oc = t.neigh_cache(pos, h, rows, 1.1)
        for precision in ("mixed", "fp64"):
            M.Tree(ctx, pos, lo, hi, level, h=h, htol=1.1)
            csr = M.neighbour_cache(ctx, rows, 1.1, precision)
            for key in ("cnt", "scanned", "entries"):
                assert np.array_equal(csr[key].cpu().numpy().view(np.uint32), oc[key]), (rows, precision, key)
    ctx.close()


@pytest.mark.parametrize("ratio", [3.0, 9.0, 11.0, 19.0, 21.0, 200.0])
def test_rows_of_wide_leaves_vs_oracle(gctx, ratio):
    """Leaves of two tight groups at opposite ends of a Morton cell, `ratio` pair radii apart."""
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(int(ratio))
    ends = np.floor(1024 * (0.1 + 0.8 * rng.random((40, 3)))) / 1024
    radius = 9e-4 / ratio
    groups = [c + np.array([[e, 4e-4, 4e-4]]) + 0.8 * radius * rng.random((12, 3))
              for c in ends for e in (1e-5, 9.5e-4 - radius)]
    pos = np.concatenate(groups + [np.array([[0.0, 0, 0], [1, 1, 1]])])
    h = np.full(len(pos), radius / 2.2) * rng.choice([1.0, 0.7], len(pos))
    lo, hi = (0.0,) * 3, (np.nextafter(1.0, 2.0),) * 3
    for level in (0, 4):
        oc = O.Tree(pos, lo, hi, level, h=h, htol=1.1).neigh_cache(pos, h, len(pos), 1.1)
        M.Tree(gctx, pos, lo, hi, level, h=h, htol=1.1)
        csr = M.neighbour_cache(gctx, len(pos), 1.1, "mixed")
        for key in ("cnt", "scanned", "entries"):
            assert np.array_equal(csr[key].cpu().numpy().view(np.uint32), oc[key]), (level, key)


def test_one_cell_is_the_work_of_many_warps(gctx):
    """20,000 particles of one cell (every row has them all as candidates): about 1 ms, and
    seconds where a leaf's rows are left to one warp."""
    import torch

    from shamrock_gb300 import modules as M

    pos, h = _clumps([20000], 9e-4, np.random.default_rng(0))
    M.Tree(gctx, pos, (0.0,) * 3, (1.0001,) * 3, 3, h=h, htol=1.1)
    best = np.inf
    for _ in range(3):
        torch.cuda.synchronize()
        t = time.perf_counter()
        gctx.call("gbsph_neighbour_cache", len(h), 1.1, 1, None)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    assert best < 0.25, best
