"""Screening sums over bins that hold several points.

A point is the mean of its cell's samples and is binned by the floor of its position, so samples
on cell faces, as a lattice gives, put the points of neighbouring cells into one bin.  The sums
take a bin's points in the order of their cells' keys, as the oracle does: bitwise the same
right-hand sides and coefficients.  The lattice is dyadic, in the unit cube as well (scale 2 about
a box of unit sides), so every mean is exact and lies on its cell's faces.
"""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _lattice(seed, count, dtype):
    rng = np.random.default_rng(seed)
    node = rng.integers(0, 9, (count, 3)) / 8.0  # corners of the depth-4 cells
    p = np.clip(np.where(rng.random((count, 3)) < 0.6, node, node + rng.integers(1, 512, (count, 3)) / 4096.0), 0, 1)
    p[0], p[1] = 0, 1
    n = rng.normal(size=(count, 3))
    return p.astype(dtype), (n / np.linalg.norm(n, axis=1)[:, None]).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("seed,count", [(0, 200), (1, 600), (3, 600)])
def test_points_on_cell_faces_sum_in_the_oracle_s_order(dtype, seed, count):
    from warp_psr_b200 import reconstruct
    p, n = _lattice(seed, count, dtype)
    opts = dict(depth=6, full_depth=3, scale=2.0, point_weight=4.0, samples_per_node=1e-8)
    r = reconstruct(torch.from_numpy(p).cuda(), torch.from_numpy(n).cuda(), keep_stages=True, **opts)
    ref = oracle.OracleResult(p, n, **opts)
    torch_dtype = torch.float64 if dtype == np.float64 else torch.float32
    for d in range(3, 7):
        np.testing.assert_array_equal(r.diagnostics["stage"](f"rhs_{d}", torch_dtype).cpu().numpy(),
                                      ref.stage(f"rhs_{d}", dtype))
    np.testing.assert_array_equal(r.field.keys.cpu().numpy(), ref.keys)
    np.testing.assert_array_equal(r.field.coefficients.cpu().numpy(), ref.coefficients)
