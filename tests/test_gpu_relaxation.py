"""Ordered sliced Gauss-Seidel: CUDA (dependency-scheduled) vs the oracle's sequential order.

Bitwise equality, as warp-psr requires of its wavefront graphs
(tests/test_relaxation.py:110-147).
"""
import numpy as np
import pytest
import torch

import oracle
from relax_cases import local_system

pytestmark = pytest.mark.gpu


def gpu_relax(keys, offsets, columns, values, b, x, depth, iters):
    from warp_psr_b200 import ops
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    xx = t(x)
    ops.relax_sliced(t(keys), depth, t(offsets), t(columns), t(values), t(b), xx, iters)
    return xx.cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("iters", [0, 1, 3, 8])
@pytest.mark.parametrize("pattern", ["full", "sparse", "empty_slices"])
def test_matches_serialized_updates_for_arbitrary_local_matrices(dtype, iters, pattern):
    keys, offsets, columns, values, b, x = local_system(pattern, dtype=dtype)
    expected = oracle.relax_sliced(keys, 3, offsets, columns, values, b, x, iters)
    actual = gpu_relax(keys, offsets, columns, values, b, x, 3, iters)
    np.testing.assert_array_equal(actual, expected)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("seed", [0, 1])
def test_many_concurrent_slices(dtype, seed):
    # 33^3 nodes at depth 5: 33 slices x 8 visits keep the whole persistent grid busy.
    keys, offsets, columns, values, b, x = local_system("random", size=33, depth=5, dtype=dtype, seed=seed)
    expected = oracle.relax_sliced(keys, 5, offsets, columns, values, b, x, 8)
    actual = gpu_relax(keys, offsets, columns, values, b, x, 5, 8)
    np.testing.assert_array_equal(actual, expected)


def test_repeated_calls_are_deterministic():
    keys, offsets, columns, values, b, x = local_system("full", size=17, depth=4, dtype=np.float32)
    first = gpu_relax(keys, offsets, columns, values, b, x, 4, 8)
    for _ in range(3):
        np.testing.assert_array_equal(gpu_relax(keys, offsets, columns, values, b, x, 4, 8), first)


def test_rejects_rows_wider_than_the_stencil():
    from warp_psr_b200 import ops
    keys, offsets, columns, values, b, x = local_system("full", dtype=np.float32)
    bad = columns.copy()
    bad[0] = len(keys) + 5
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    with pytest.raises(ValueError, match="out of range"):
        ops.relax_sliced(t(keys), 3, t(offsets), t(bad), t(values), t(b), t(x), 2)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows", [1, 2, 31, 33, 257, 729])
def test_rows_with_any_of_their_entries_missing(dtype, rows):
    # the first `rows` rows of a full level, entries dropped at random (diagonals among them:
    # such rows are not updated), a row emptied; bitwise against the sequential order
    keys, offsets, columns, values, b, x = local_system("full", dtype=dtype)
    rng = np.random.default_rng(rows)
    new_off, cols, vals = [0], [], []
    for i in range(rows):
        e = np.arange(offsets[i], offsets[i + 1])
        keep = (columns[e] < rows) & (rng.random(len(e)) < 0.8) & (i != rows // 2)
        cols.append(columns[e[keep]])
        vals.append(values[e[keep]])
        new_off.append(new_off[-1] + int(keep.sum()))
    cols, vals = np.concatenate(cols), np.concatenate(vals)
    if not len(cols):  # the library takes no empty arrays: one entry past the last row
        cols, vals = np.zeros(1, np.int32), np.ones(1, dtype)
    off = np.array(new_off, np.int32)
    expected = oracle.relax_sliced(keys[:rows], 3, off, cols, vals, b[:rows], x[:rows], 3)
    actual = gpu_relax(keys[:rows], off, cols, vals, b[:rows], x[:rows], 3, 3)
    np.testing.assert_array_equal(actual, expected)


@pytest.mark.parametrize("fault,message", [("order", "ascending"), ("repeat", "ascending"), ("far", "neighbourhood"),
                                           ("wide", "27 entries"), ("negative", "out of range"),
                                           ("depth", "basis keys"), ("outside", "basis keys")])
def test_rejected_rows_name_their_fault(fault, message):
    from warp_psr_b200 import ops
    keys, offsets, columns, values, b, x = local_system("full", dtype=np.float32)
    r = len(keys) // 2
    e = offsets[r]
    if fault == "order":
        columns[e], columns[e + 1] = columns[e + 1], columns[e]
    elif fault == "repeat":
        columns[e + 1] = columns[e]
    elif fault == "far":
        columns[offsets[0]] = len(keys) - 1
    elif fault == "wide":
        offsets[r] -= 5
    elif fault == "negative":
        columns[e] = -1
    elif fault == "depth":
        keys = keys + (1 << 48)
    elif fault == "outside":
        keys = np.sort(keys + 5)  # every z moved up: the last five slices leave the grid
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    with pytest.raises(ValueError, match=message):
        ops.relax_sliced(t(keys), 3, t(offsets), t(columns), t(values), t(b), t(x), 2)
