"""Ordering of a build's triples by output row (order_rows, order_rows_long):
rows of one warp (64 triples), of a block's tile (2048) and longer, mixed in
one block of 32 rows and across blocks, against the oracle bit for bit."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def graded(parts, angle):
    """A grid over [-1, 1]^2 whose lines lie at the given fractions, turned a little."""
    t = -0.97 + 1.94 * np.asarray(parts)
    y, x = np.meshgrid(t, t, indexing="ij")
    return np.stack([x * np.cos(angle) - y * np.sin(angle), x * np.sin(angle) + y * np.cos(angle)])


@pytest.mark.parametrize(
    "n_in, parts",
    [
        (9, np.linspace(0, 1, 4)),  # one block, short rows
        (12, np.linspace(0, 1, 34)),  # 33^2 rows: a last block of one row
        (75, np.linspace(0, 1, 2)),  # one row, longer than two tiles
        (60, np.r_[0, 0.7, 0.71, 0.72, 0.75, 0.8, 1]),  # long and short rows in a block
        (40, np.r_[0, 0.5, np.linspace(0.52, 1, 40)]),  # blocks with and without long rows
        (20, np.linspace(0, 1, 6)),  # rows around 64 triples
    ],
)
def test_rows_of_every_length(n_in, parts):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import regridding_gb300 as rg

    gi = graded(np.linspace(0, 1, n_in + 1) ** 1.1, 0.013) * 1.05
    go = graded(parts, -0.021)
    want = oracle.weights_conservative_2d(gi, go)
    got = rg.build_conservative_2d(gi, go).export_numpy()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize(
    "scale", [(1.0, 2.0**-385), (1.0, 2.0**-393), (1.0, 2.0**-420), (2.0**60, 2.0**345), (1e60, 1e61), (1e70, 1e70)]
)
def test_weights_at_any_scale(scale):
    """area / cell area beside the limits 2^-400 and 2^400 of area_ratio's short form"""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import regridding_gb300 as rg

    scale = np.reshape(scale, (2, 1, 1))
    gi = graded(np.linspace(0, 1, 24) ** 1.1, 0.013) * 1.05 * scale
    go = graded(np.linspace(0, 1, 18), -0.021) * scale
    want = oracle.weights_conservative_2d(gi, go)
    got = rg.build_conservative_2d(gi, go).export_numpy()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_long_rows_side_by_side():
    """A coarse pair whose 64 rows have some 36,000 triples each takes about as
    long beside 63 fine pairs, where they lie in two blocks of 32 rows, as
    alone, where each pair of rows has a block (in series they took ten times
    as long)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import time

    from regridding_gb300 import batching, workloads

    def device(grid):
        return tuple(torch.tensor(np.asarray(a), device="cuda") for a in grid)

    gi = np.stack(np.meshgrid(np.linspace(0, 1, 513), np.linspace(0, 1, 513), indexing="ij"))
    go = np.stack(np.meshgrid(np.linspace(0.013, 0.977, 9), np.linspace(0.013, 0.977, 9), indexing="ij"))
    coarse = device(gi + 1e-4 * np.sin(40 * gi[::-1])), device(go + 1e-7 * np.sin(9 * go[::-1]))
    rng = np.random.default_rng(2)
    fine = [tuple(device(g) for g in workloads.grid_pair(rng, 64)) for _ in range(63)]
    seconds = []
    for pairs in ([coarse], fine + [coarse]):
        times = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            built = batching.build_batch(pairs)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
            last = built[-1].export_numpy()
            for dw in built:
                dw.free()
        seconds.append((min(times), last))
    assert all(np.array_equal(a, b) for a, b in zip(seconds[0][1], seconds[1][1]))
    assert seconds[1][0] < 3 * seconds[0][0], [t for t, _ in seconds]
