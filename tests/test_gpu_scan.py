"""Builds whose scans over the output rows take one tile (4,096 elements), the
most tiles that two kernels take (1,024), and one more, against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, columns", [(63, 65), (64, 64), (1023, 4100), (1024, 4096)])
def test_rows_on_both_sides_of_a_tile_count(rows, columns):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import regridding_gb300 as rg

    t = np.linspace(-1.03, 1.01, 4)
    y, x = np.meshgrid(t, t, indexing="ij")
    gi = np.stack([x + 0.11 * y, y - 0.07 * x])
    v, u = np.meshgrid(np.linspace(-0.9, 0.91, rows + 1), np.linspace(-0.92, 0.9, columns + 1), indexing="ij")
    go = np.stack([u, v])
    want = oracle.weights_conservative_2d(gi, go)
    got = rg.build_conservative_2d(gi, go).export_numpy()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
