"""Morton codes in boxes without extent along an axis, unbounded boxes and boxes at the ends
of the double range, where the grid quotient can be 0 / 0 or inf / inf."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = np.inf
BOXES = [((0, 0, 0.5), (1, 1, 0.5)), ((0.5,) * 3, (0.5,) * 3), ((0, 0, 0), (0, 0, 0)), ((1, 1, 1), (0, 0, 0)),
         ((0, 0, 0), (INF, 1, 1)), ((-INF, 0, 0), (1, 1, 1)), ((0, 0, 0), (1e-320, 1e-310, 1)),
         ((-1.7e308, 0, 0), (1.7e308, 1e308, 1)), ((0, 0, 0), (1, 1, 1))]


def _codes(pos, lo, hi, bits):
    """min(trunc(quotient), top) interleaved, the top cell where the quotient is no number."""
    top = (1 << bits) - 1
    lo, hi = np.array(lo, float), np.array(hi, float)
    with np.errstate(all="ignore"):
        step = (hi - lo) / float(1 << bits)
        q = (np.fmin(np.fmax(pos, lo), hi) - lo) / step
    cell = np.where(np.isnan(q), top, np.clip(np.nan_to_num(q, nan=0, posinf=top, neginf=0), 0, top)).astype(np.uint64)
    out = np.zeros(len(pos), np.uint64)
    for b in range(bits):
        for c in range(3):
            out |= ((cell[:, c] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - c)
    return out


@pytest.mark.parametrize("key_bits,bits", [(32, 10), (64, 21)])
@pytest.mark.parametrize("box", BOXES)
def test_cells_without_a_quotient(gctx, key_bits, bits, box):
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(0)
    pos = np.concatenate([rng.random((40, 3)), [[0.5, 0.5, 0.5], [0, 0.7, 1], [np.nan, 0.5, 0.5], [INF, 0.1, -INF],
                                                [0.25, 0.5, 0.5], [1, 1, 1]]])
    got = M.unsigned(M.morton_codes(gctx, pos, *box, key_bits=key_bits), key_bits).astype(np.uint64)
    assert np.array_equal(got, _codes(pos, *box, bits))


def test_planar_tree_vs_its_codes(gctx):
    """A tree over particles of one plane, in the box that holds them exactly."""
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(1)
    pos = rng.random((500, 3))
    pos[:, 2] = 0.5
    lo, hi = pos.min(0), pos.max(0)
    e = M.Tree(gctx, pos, lo, hi, 0).export()
    assert np.array_equal(np.asarray(e["sorted_keys"][:500], np.uint64), np.sort(_codes(pos, lo, hi, 10)))
