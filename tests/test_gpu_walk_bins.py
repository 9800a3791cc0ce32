"""Walk steps outside the static grid: the boundary bins chosen in float32
(boundary_bins), or in FP64 where an offset makes float32 too coarse, give the
oracle's weights bit for bit.  The bent boundary lets lines leave and enter
several times."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def bent(n, extent, amp, offset):
    t = np.linspace(-extent, extent, n + 1)
    y, x = np.meshgrid(t, t, indexing="ij")
    c, s = np.cos(0.37), np.sin(0.37)
    u, v = x * c - y * s, x * s + y * c
    return np.stack([u + amp * np.sin(4 * v), v + amp * np.sin(3 * u)]) + offset


@pytest.mark.parametrize("offset", [0.0, 40.0, -3e3, 2e5])
@pytest.mark.parametrize("n_in, n_out", [(48, 31), (5, 60)])
def test_lines_across_the_boundary(n_in, n_out, offset):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import regridding_gb300 as rg

    gi = bent(n_in, 1.0, 0.09, offset)
    go = bent(n_out, 1.31, 0.0, offset)[::-1, ::-1] + np.reshape([0.0137, -0.0071], (2, 1, 1))
    want = oracle.weights_conservative_2d(gi, go)
    got = rg.build_conservative_2d(gi, go).export_numpy()
    assert len(want[0]) > 0
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
