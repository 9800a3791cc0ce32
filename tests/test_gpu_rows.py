"""1D weights of many rows on the GPU: the merge of the sweep and the block
diagonal apply against the oracle's element by element."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def rows(case, rng):
    """(x_in, x_out) of a few rows."""
    if case == "shifted":
        x, y = np.linspace(0, 1, 30) + rng.uniform(-0.6, 0.6, (9, 1)), np.linspace(0, 1, 23) + np.zeros((9, 1))
    elif case == "apart":
        x, y = np.linspace(0, 1, 5) + np.zeros((4, 1)), np.linspace(0, 1, 7) + np.array([[1.0], [-1.0], [2.0], [-3.0]])
    elif case == "shared":  # vertices of both grids
        x, y = np.arange(0, 41.0) + np.zeros((5, 1)), np.arange(-8, 60.0, 1) / 2 + np.array([[0], [1], [8], [36], [-17.5]])
    elif case == "same":
        x = np.sort(rng.uniform(0, 1, (3, 300)), axis=1)
        y = x.copy()
    elif case == "smallest":
        x, y = np.sort(rng.uniform(0, 1, (6, 2)), axis=1), np.sort(rng.uniform(0, 1, (6, 2)), axis=1)
    elif case == "blocks":  # more vertices than threads of a block
        x, y = np.sort(rng.uniform(0, 1, (2, 1023)), axis=1), np.sort(rng.uniform(-0.1, 1.1, (2, 513)), axis=1)
    elif case == "ranks":  # static vertices on both sides of what shared memory holds
        return np.sort(rng.uniform(0, 1, (1, 700)), axis=1), np.sort(rng.uniform(0, 1, (1, 8192 + 3)), axis=1)
    else:  # "uneven": repeated and falling steps
        x, y = np.linspace(0, 1, 20) + np.zeros((4, 1)), np.linspace(-0.1, 1.1, 15) + np.zeros((4, 1))
        x[0, 7] = x[0, 6]
        y[1, 5] = y[1, 4]
        x[2, 9] = 0.1
        y[3, 6] = 0.9
    return x, y


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("flip", ["", "x", "y", "xy"])
@pytest.mark.parametrize("case", ["shifted", "apart", "shared", "same", "smallest", "blocks", "ranks", "uneven"])
def test_conservative_rows_match_oracle(case, flip, weighted):
    import regridding_gb300 as rg

    rng = np.random.default_rng(3)
    x, y = rows(case, rng)
    x = x[:, ::-1] if "x" in flip else x
    y = y[:, ::-1] if "y" in flip else y
    w_in = rng.normal(0, 1, (x.shape[0], x.shape[1] - 1)) if weighted else None
    got, *_ = rg.weights((x,), (y,), axis_input=-1, axis_output=-1, weights_input=w_in, method="conservative")
    v = rng.normal(0, 1, (x.shape[0], x.shape[1] - 1))
    out = None
    if not weighted:
        out = rg.regrid((x,), (y,), v, axis_input=-1, axis_output=-1, method="conservative")
    for d in range(x.shape[0]):
        ii, oo, vv = oracle.coalesce(*oracle.conservative_1d(x[d], y[d], None if w_in is None else w_in[d]))
        for a, b in zip(got[d], (ii, oo, vv)):
            np.testing.assert_array_equal(a, b)
        if out is not None:
            want = oracle.apply(ii, oo, vv, v[d:d + 1], y.shape[1] - 1)[0]
            np.testing.assert_array_equal(out[d], want)


@pytest.mark.parametrize("method", ["conservative", "multilinear"])
@pytest.mark.parametrize("lead", [(), (3,)])
@pytest.mark.parametrize("axis", [-1, -2])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_rows_equal_elements(method, lead, axis, dtype):
    """regrid of rows with their own grids, regrid_from_weights of their saved
    weights, and each element alone: the same bits."""
    import regridding_gb300 as rg

    rng = np.random.default_rng(4)
    edges = int(method == "conservative")
    x = np.sort(rng.uniform(0, 1, (6, 12 + edges)), axis=1)
    y = np.sort(rng.uniform(0, 1, (6, 9 + edges)), axis=1)
    v = rng.normal(0, 1, lead + (6, 12)).astype(dtype)
    if axis == -2:
        x, y, v = x.T, y.T, np.swapaxes(v, -1, -2)
    kw = {"axis_input": axis, "axis_output": axis}
    out = rg.regrid((x,), (y,), v, method=method, **kw)
    saved = rg.weights((x,), (y,), method=method, **kw)
    np.testing.assert_array_equal(out, rg.regrid_from_weights(*saved, v, **kw))
    into = np.zeros(out.shape, dtype="float32")
    rg.regrid((x,), (y,), v, values_output=into, method=method, **kw)
    for d in range(6):
        pick = (lambda a: a[d]) if axis == -1 else (lambda a: a[:, d])
        one = rg.weights((np.ascontiguousarray(pick(x)),), (np.ascontiguousarray(pick(y)),), method=method)
        vd = v[..., d, :] if axis == -1 else v[..., d]
        want = rg.regrid_from_weights(*one, vd, axis_input=-1, axis_output=-1)
        got = out[..., d, :] if axis == -1 else out[..., d]
        np.testing.assert_array_equal(got, want)
        w32 = np.zeros(want.shape, dtype="float32")
        rg.regrid_from_weights(*one, vd, values_output=w32, axis_input=-1, axis_output=-1)
        np.testing.assert_array_equal(into[..., d, :] if axis == -1 else into[..., d], w32)


@pytest.mark.parametrize("flip", ["", "x", "y", "xy"])
def test_many_rows_equal_few(flip):
    """30,000 short rows at a time, every third with a repeated or falling
    step, and a hundred of them alone: the same bits."""
    import regridding_gb300 as rg

    rng = np.random.default_rng(11)
    x = np.sort(rng.uniform(0, 1, (30_000, 34)), axis=1)
    y = np.sort(rng.uniform(-0.1, 1.1, (30_000, 27)), axis=1)
    x[::3, 7] = x[::3, 6]
    y[1::9, 5] = y[1::9, 4]
    x[2::27, 9] = x[2::27, 5]
    x = x[:, ::-1] if "x" in flip else x
    y = y[:, ::-1] if "y" in flip else y
    many, *_ = rg.weights((x,), (y,), axis_input=-1, axis_output=-1, method="conservative")
    for k in (0, 1, 2, 15_000, 29_900):
        few, *_ = rg.weights((x[k:k + 100],), (y[k:k + 100],), axis_input=-1, axis_output=-1, method="conservative")
        for a, b in zip(few, many[k:k + 100]):
            for p, q in zip(a, b):
                np.testing.assert_array_equal(p, q)


def test_uneven_rows_take_no_longer():
    """10,000 rows with a repeated vertex take about as long as without (a
    block for each row's one sweeping thread made them ten times slower)."""
    import time

    import torch

    from regridding_gb300 import _device, _lib

    nd, m, n = 10_000, 513, 385
    cap = m + n + 2
    y = torch.linspace(-0.05, 1.05, n, dtype=torch.float64, device="cuda").repeat(nd, 1)
    x = torch.sort(torch.rand(nd, m, dtype=torch.float64, device="cuda"), dim=1).values
    ii, oo = (torch.empty(nd, cap, dtype=torch.int64, device="cuda") for _ in range(2))
    vv, count = torch.empty(nd, cap, dtype=torch.float64, device="cuda"), torch.empty(nd, dtype=torch.int64, device="cuda")
    seconds = []
    for uneven in (False, True):
        if uneven:
            x[:, m // 2] = x[:, m // 2 - 1]
        times = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            _lib.call("rg_conservative_1d", _device.ptr(x), m, m, _device.ptr(y), n, n, nd, None, 0, cap,
                      _device.ptr(ii), _device.ptr(oo), _device.ptr(vv), _device.ptr(count), _device.stream())
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        seconds.append(min(times))
    assert seconds[1] < 3 * seconds[0], seconds
