"""Routes that a rule on sizes chooses, on both sides of the rule."""
import numpy as np
import pytest

from test_gpu_step import make_pair

pytestmark = pytest.mark.gpu


def _lattice_state(nx, ny, nz, ties, seed=0):
    """A jittered lattice (no two particles in a Morton cell of 1/1024 of the box) and
    `ties` close pairs that share one."""
    rng = np.random.default_rng(seed)
    d = 1.0 / max(nx, ny, nz)
    pos = np.stack(np.meshgrid(*[(np.arange(k) + 0.5) * d for k in (nx, ny, nz)], indexing="ij"), -1).reshape(-1, 3)
    pos = pos + 0.1 * d * (rng.random(pos.shape) - 0.5)
    pick = rng.choice(len(pos), ties, replace=False)
    pos = np.concatenate([pos, pos[pick] + 1e-7 * rng.standard_normal((ties, 3))])
    n = len(pos)
    return dict(pos=pos, vel=np.zeros((n, 3)), h=np.full(n, 1.2 * d), u=np.ones(n), gamma=1.4, pmass=1.0 / n,
                box_min=(0, 0, 0), box_max=(1, 1, 1))


@pytest.mark.parametrize("shape,ties", [((2, 1, 1), 0), ((13, 9, 7), 0), ((13, 9, 7), 5), ((128, 128, 64), 0),
                                        ((102, 102, 101), 0), ((102, 102, 101), 40)])
def test_step_sort_is_the_networks(shape, ties):
    """The permutation after a step equals the bitonic network's over the same keys, by the
    network itself (up to 2^20 keys), the radix sort, and the radix sort's fall-back."""
    from shamrock_gb300 import modules as M

    model, _ = make_pair(_lattice_state(*shape, ties), precision="mixed", periodic=False)
    model.set_next_dt(0.0)
    model.evolve_once()
    import ctypes as C
    import torch

    ctx = model._lib_ctx
    P, Lc = C.c_uint32(), C.c_uint32()
    ctx.call("gbsph_tree_counts", C.byref(P), C.byref(Lc))
    keys = torch.empty(P.value, dtype=torch.int32, device="cuda")
    perm = torch.empty(P.value, dtype=torch.int32, device="cuda")
    ctx.call("gbsph_tree_export", C.c_void_p(keys.data_ptr()), C.c_void_p(perm.data_ptr()), *([None] * 11))
    torch.cuda.synchronize()
    unsorted = torch.empty_like(keys)
    unsorted[perm.long()] = keys
    want_keys, want = M.sort_by_key(ctx, unsorted, key_bits=32)
    assert torch.equal(keys, want_keys)
    n = len(model.collect_data()["hpart"])
    assert torch.equal(perm[:n], want[:n])
    assert (len(torch.unique(keys[:n])) < n) == (ties > 0)


@pytest.mark.parametrize("n", [1, 2, 9, 513, 40000, 60000])
def test_cache_routes_vs_oracle(gctx, n):
    """Stage 1 on the wide hierarchy (up to 320 owning leaves an SM) and on the binary tree, one
    leaf per particle, with a clump of small h far from the origin (rows decided in FP64)
    and rows longer than the 64 candidates that stage 2 tests at a time."""
    from oracle import oracle as O
    from shamrock_gb300 import modules as M

    rng = np.random.default_rng(n)
    pos = 5.0 + rng.random((n, 3))
    h = rng.uniform(0.5, 1.1, n) * (30.0 / max(n, 30)) ** (1 / 3) * 0.5
    k = n // 10
    pos[:k] = 5.5 + 1e-4 * rng.standard_normal((k, 3))
    h[:k] = 3e-5
    lo, hi = np.nextafter(pos.min(0), -np.inf), np.nextafter(pos.max(0), np.inf)
    M.Tree(gctx, pos, lo, hi, 0, h=h, htol=1.1)
    csr = M.neighbour_cache(gctx, n, 1.1, "mixed")
    o = O.Tree(pos, lo, hi, 0, h=h, htol=1.1)
    oc = o.neigh_cache(pos, h, n, 1.1)
    for key in ("cnt", "scanned", "entries"):
        assert np.array_equal(csr[key].cpu().numpy().view(np.uint32), oc[key]), key


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 7, 3), (32, 32, _sms() // 4), (32, 32, _sms() // 4 + 1)])
def test_row_routes_mixed_vs_fp64(shape):
    """Mixed step with four lanes per row (up to 256 rows an SM) and a thread per row in the
    density passes, four lanes in the derivatives, free boundary (rows of every length):
    within the tier's 1e-5 of the FP64 step from the same state."""
    s = _lattice_state(*shape, 0, seed=3)
    out = []
    for precision in ("mixed", "fp64"):
        model, _ = make_pair(s, precision=precision, periodic=False)
        model.set_next_dt(0.0)
        model.evolve_once()
        out.append(model.collect_data())
    for key in ("hpart", "omega", "axyz", "duint"):
        a, b = out[0][key], out[1][key]
        assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-300), key


def test_cache_overflowing_lists_vs_oracle():
    """Stage-1 lists and rows longer than their slots in a new context: stage 2 has then run
    over cut lists and both stages run again; the next build has the slots."""
    from oracle import oracle as O
    from shamrock_gb300 import _lib, modules as M

    rng = np.random.default_rng(8)
    n = 2000
    pos = rng.random((n, 3))
    h = np.where(rng.random(n) < 0.5, 0.6, 0.01)
    lo, hi = np.nextafter(pos.min(0), -np.inf), np.nextafter(pos.max(0), np.inf)
    oc = O.Tree(pos, lo, hi, 0, h=h, htol=1.1).neigh_cache(pos, h, n, 1.1)
    ctx = _lib.Context(0)
    for _ in range(2):
        M.Tree(ctx, pos, lo, hi, 0, h=h, htol=1.1)
        csr = M.neighbour_cache(ctx, n, 1.1, "mixed")
        for key in ("cnt", "scanned", "entries"):
            assert np.array_equal(csr[key].cpu().numpy().view(np.uint32), oc[key]), key
