"""The tree built on bitmaps (depths through 11) against the tree built by sorting (PSR_TREE=sort,
the path of deeper trees): the same support and basis keys, in the same order, for every
relation of base, full and finest depth."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cloud(count, seed):
    rng = np.random.default_rng(seed)
    n = rng.normal(size=(count, 3))
    n /= np.linalg.norm(n, axis=1)[:, None]
    p = n * (1 + 0.2 * n[:, :1]) + 0.05 * rng.normal(size=(count, 3))
    return torch.from_numpy(p).cuda(), torch.from_numpy(n).cuda()


@pytest.mark.parametrize("depth,full_depth,base_depth", [(1, 0, 0), (1, 1, 1), (2, 1, 0), (3, 3, 3), (4, 2, 0),
                                                         (5, 4, 3), (5, 5, 4), (6, 3, 3), (6, 5, 2), (7, 6, 6),
                                                         (8, 4, 4), (9, 3, 1), (11, 2, 2)])
@pytest.mark.parametrize("count", [5, 3000])
def test_bitmap_tree_has_the_sorted_tree_s_keys(monkeypatch, depth, full_depth, base_depth, count):
    from warp_psr_b200 import reconstruct
    P, N = _cloud(count, seed=depth)
    runs = []
    for mode in (None, "sort"):
        if mode:
            monkeypatch.setenv("PSR_TREE", mode)
        r = reconstruct(P, N, depth=depth, full_depth=full_depth, base_depth=base_depth, iters=1, scale=1.1)
        runs.append((r.field.keys.cpu().numpy(), [k.cpu().numpy()
                                                  for k in r.diagnostics["support_keys"]]))
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    assert len(runs[0][1]) == len(runs[1][1]) == depth + 1
    for a, b in zip(runs[0][1], runs[1][1]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("depth,full_depth", [(10, 2), (11, 2), (12, 1)])
def test_deep_records_match_the_oracle(dtype, depth, full_depth):
    """32-bit record keys through depth 10 and 64-bit ones beyond, bitmap trees through depth 11
    and sorted ones beyond: every basis key, and the density and normal fields behind them."""
    import oracle
    from warp_psr_b200 import reconstruct
    P, N = _cloud(200, seed=depth)
    p, n = P.cpu().numpy().astype(dtype), N.cpu().numpy().astype(dtype)
    opts = dict(depth=depth, full_depth=full_depth, base_depth=1, iters=1, samples_per_node=1e-8)  # finest records
    r = reconstruct(torch.from_numpy(p).cuda(), torch.from_numpy(n).cuda(), **opts)
    ref = oracle.OracleResult(p, n, **opts)
    np.testing.assert_array_equal(r.field.keys.cpu().numpy(), ref.keys)
    tol = 2e-6 if dtype == np.float32 else 1e-13  # per stage, and 8 times it on the coefficients
    scale = np.abs(ref.coefficients).max()
    assert np.abs(r.field.coefficients.cpu().numpy() - ref.coefficients).max() <= 8 * tol * scale


@pytest.mark.parametrize("count,finest", [(5, 3), (3000, 7)])
def test_bitmaps_reach_down_to_the_finest_records_only(count, finest):
    """A sparse cloud at depth 11: no record lies deeper than `finest`, so the tree needs none of
    the 321 MB of bitmaps and counts of the levels below (459 MB at the peak with them, of which
    the dense column tables of the basis keys and the records take 85)."""
    import ctypes
    from warp_psr_b200 import _lib, reconstruct
    _lib.load()
    rt = ctypes.CDLL("libcudart.so.12")
    pool, used_high, word = ctypes.c_void_p(), 8, ctypes.c_uint64(0)  # cudaMemPoolAttrUsedMemHigh
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    P, N = _cloud(count, seed=11)
    torch.cuda.synchronize()
    assert rt.cudaMemPoolSetAttribute(pool, used_high, ctypes.byref(word)) == 0
    r = reconstruct(P, N, depth=11, full_depth=2, solve_depth=2, keep_stages=True)
    torch.cuda.synchronize()
    assert rt.cudaMemPoolGetAttribute(pool, used_high, ctypes.byref(word)) == 0
    assert int(r.diagnostics["stage"]("normal_keys", torch.int64).max()) >> 48 <= finest
    assert word.value < 200 << 20
