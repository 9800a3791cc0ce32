"""The float32 decision of point-in-cell tests on the GPU: points on, and at
every distance from, the edges and vertices of the cells, against the oracle's
FP64 tests."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0.0, 3.0, 1e4, 1e9])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-14, 1e-30, 1e20, 1e200])
@pytest.mark.parametrize("grid", ["regular", "bent", "flipped"])
def test_points_near_edges(grid, scale, offset):
    import regridding_gb300 as rg

    rng = np.random.default_rng(8)
    x, y = np.meshgrid(np.linspace(-1, 1, 9), np.linspace(-1, 1, 7), indexing="ij")
    if grid != "regular":
        x, y = 0.9 * x - 0.4 * y, 0.4 * x + 0.9 * y
        x, y = x + 0.05 * np.sin(3 * y), y + 0.05 * np.sin(3 * x)
    if grid == "flipped":
        x, y = x[::-1], y[::-1]
    g = tuple(np.ascontiguousarray(c * scale + offset * scale) for c in (x, y))
    a = (g[0][:-1].ravel(), g[1][:-1].ravel())
    b = (g[0][1:].ravel(), g[1][1:].ravel())
    c = (g[0][:, 1:].ravel(), g[1][:, 1:].ravel())
    d = (g[0][:, :-1].ravel(), g[1][:, :-1].ravel())
    px, py = [], []
    for p, q in ((a, b), (d, c)):
        t = rng.choice([0.0, 1.0, 0.5, 0.25, 0.3, 0.77], p[0].size)
        for away in (0.0, 1e-17, 1e-12, 1e-8, 3e-7, 1e-5, 1e-2):
            for sign in (-1, 1):
                nx, ny = q[1] - p[1], p[0] - q[0]
                px.append(p[0] + t * (q[0] - p[0]) + sign * away * nx)
                py.append(p[1] + t * (q[1] - p[1]) + sign * away * ny)
    px, py = np.concatenate(px), np.concatenate(py)
    px[:3], py[3:6] = np.nan, np.inf
    want = oracle.locate(g, px, py, "brute")
    got = rg.locate_2d(g, px, py, method="exhaustive")
    for u, v in zip(got, want):
        np.testing.assert_array_equal(u, v)
    # the grid walk and the secant iteration say nothing of points that are no
    # numbers, nor the walk of coordinates whose products overflow
    fine = np.isfinite(px) & np.isfinite(py)
    for method in ("brute", "secant") if scale < 1e100 else ("secant",):
        got = rg.locate_2d(g, px[fine], py[fine], method=method)
        for u, v in zip(got, oracle.locate(g, px[fine], py[fine], method)):
            np.testing.assert_array_equal(u, v)
