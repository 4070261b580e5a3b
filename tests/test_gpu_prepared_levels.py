"""Levels prepared ahead of the chain, on a stream of their own, and levels prepared when the chain
reaches them: the same results, and the peak memory of one level at a time where none is prepared
ahead (PSR_AHEAD_BYTES bounds what the levels prepared ahead may hold: none, some of them, all).  A
call that runs out of memory with levels held together is solved again one level at a time
(PSR_AHEAD_FAIL makes the preparation ahead of a level report that, on the host)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cloud(count, dtype, seed=3):
    rng = np.random.default_rng(seed)
    n = rng.normal(size=(count, 3))
    n /= np.linalg.norm(n, axis=1)[:, None]
    p = n * (1 + 0.2 * n[:, :1]) + 0.02 * rng.normal(size=(count, 3))
    return torch.from_numpy(p.astype(dtype)).cuda(), torch.from_numpy(n.astype(dtype)).cuda()


@pytest.mark.parametrize("dtype,precision", [(np.float32, "input"), (np.float64, "input"), (np.float32, "mixed")])
@pytest.mark.parametrize("point_weight", [0.0, 2.0])
@pytest.mark.parametrize("bound", ["0", "300000", "3000000"])
def test_results_do_not_depend_on_the_levels_prepared_ahead(monkeypatch, dtype, precision, point_weight, bound):
    from warp_psr_b200 import reconstruct, reconstruct_differentiable
    P, N = _cloud(4000, dtype)
    opts = dict(depth=6, full_depth=2, base_depth=1, precision=precision, point_weight=point_weight)
    runs = []
    for value in (None, bound):
        if value is not None:
            monkeypatch.setenv("PSR_AHEAD_BYTES", value)
        plain = reconstruct(P, N, **opts)
        taped = reconstruct_differentiable(P.clone().requires_grad_(True), N, **opts)
        runs.append([plain.field.coefficients, plain.field.cumulative, taped.coefficients.detach()])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    assert torch.equal(runs[0][0], runs[0][2])


def test_short_memory_holds_one_level_at_a_time(monkeypatch):
    """5,000 points with a chain of nodes down to depth 9 each: five levels of about the same size
    (492 MB one level at a time, 713 MB with all of them prepared ahead)."""
    from warp_psr_b200 import _lib, reconstruct
    _lib.load()
    rt = ctypes.CDLL("libcudart.so.12")
    pool, used_high = ctypes.c_void_p(), 8  # cudaMemPoolAttrUsedMemHigh
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    P, N = _cloud(5000, np.float32)
    peaks = []
    for bound in (str(1 << 40), "0"):
        monkeypatch.setenv("PSR_AHEAD_BYTES", bound)
        word = ctypes.c_uint64(0)
        torch.cuda.synchronize()
        assert rt.cudaMemPoolSetAttribute(pool, used_high, ctypes.byref(word)) == 0
        reconstruct(P, N, depth=9, full_depth=3, samples_per_node=1e-8)
        torch.cuda.synchronize()
        assert rt.cudaMemPoolGetAttribute(pool, used_high, ctypes.byref(word)) == 0
        peaks.append(word.value)
    assert peaks[1] < 0.8 * peaks[0]


@pytest.mark.parametrize("dtype,precision", [(np.float32, "input"), (np.float32, "mixed")])
@pytest.mark.parametrize("level", [2, 4, 6])
def test_running_out_of_memory_ahead_solves_one_level_at_a_time(monkeypatch, dtype, precision, level):
    from warp_psr_b200 import reconstruct, reconstruct_differentiable
    P, N = _cloud(4000, dtype)
    opts = dict(depth=6, full_depth=2, base_depth=1, precision=precision)
    torch_dtype = torch.float64 if precision == "mixed" else torch.float32
    runs = []
    for value in (None, str(level)):
        if value is not None:
            monkeypatch.setenv("PSR_AHEAD_FAIL", value)
        r = reconstruct(P, N, keep_stages=True, **opts)
        x = P.clone().requires_grad_(True)
        taped = reconstruct_differentiable(x, N, **opts)
        taped.iso_value.backward()
        runs.append(dict(coefficients=r.field.coefficients, taped=taped.coefficients.detach(),
                         rhs=[r.diagnostics["stage"](f"rhs_{d}", torch_dtype) for d in range(1, 7)],
                         counts=(r.diagnostics["relax_row_visits"], r.diagnostics["relax_launches"],
                                 r.diagnostics["relax_finest_row_visits"]), gradient=x.grad))
    a, b = runs
    assert torch.equal(a["coefficients"], b["coefficients"]) and torch.equal(a["taped"], b["taped"])
    assert all(torch.equal(x, y) for x, y in zip(a["rhs"], b["rhs"]))
    assert a["counts"] == b["counts"]
    # the reverse pass adds with atomics: to rounding
    bound = 1e-4 if precision == "input" else 1e-10
    assert float((a["gradient"] - b["gradient"]).abs().max()) <= bound * float(a["gradient"].abs().max())
