"""fill() by clusters of blocks against the oracle's sequential sweep: sizes
around what a block's threads keep, empty classes, odd seams, many slices,
more iterations than one launch takes."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("shape,missing,iterations", [
    ((1, 2, 2), 0.5, 3), ((1, 3, 3), 0.9, 5), ((2, 2, 5), 0.6, 4), ((3, 5, 4), 0.95, 7),
    ((1, 200, 301), 0.9, 6),     # more cells than the cluster's threads keep
    ((1, 64, 64), 0.25, 1025),   # two launches
    ((9, 31, 32), 0.3, 20), ((20, 17, 19), 0.3, 20), ((150, 16, 17), 0.4, 9), ((700, 8, 9), 0.3, 3),
    ((2, 33, 32), 0.0, 3),       # nothing missing
])
def test_clusters_match_oracle(dtype, shape, missing, iterations):
    import regridding_gb300 as rg

    rng = np.random.default_rng(shape[1] * 100 + shape[2])
    a = rng.normal(5, 3, shape).astype(dtype)
    where = rng.uniform(0, 1, shape) < missing
    where[0, 0, 0] = False
    if shape[0] > 2:
        where[1] = False       # a slice with nothing missing
        where[2, 1:] = True    # and one with nearly everything
    a[where] = np.nan
    got = rg.fill(a, axis=(-2, -1), num_iterations=iterations)
    want = oracle.fill(a, where, axis=(-2, -1), num_iterations=iterations)
    np.testing.assert_array_equal(got, want)


def test_many_slices_of_few_cells():
    """5000 slices with 1 % missing take no longer than with 8 % (by clusters,
    in eight rounds of blocks whose phases wait for barriers, they took ten
    times as long)."""
    import time

    import torch

    from regridding_gb300 import _device, _lib

    seconds = {}
    for share in (0.01, 0.08):
        gen = torch.Generator(device="cuda").manual_seed(3)
        a = torch.rand(5000, 32, 32, dtype=torch.float64, device="cuda", generator=gen) + 5
        where = (torch.rand(a.shape, device="cuda", generator=gen) < share).to(torch.uint8)
        guess = torch.full((5000,), 5.5, dtype=torch.float64, device="cuda")
        times = []
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            _lib.call("rg_fill_gauss_seidel", _device.ptr(a), _lib.RG_F64, _device.ptr(where), 5000, 32, 32,
                      _device.ptr(guess), _lib.RG_FILL_GUESS_SLICE, 100, _device.stream())
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        seconds[share] = min(times)
    assert seconds[0.01] < 2 * seconds[0.08], seconds
