"""Shapes set on handles that applies have already used."""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def handle(shape_in, shape_out):
    """A handle from saved entries, its sums in numpy and stacks for it."""
    torch = pytest.importorskip("torch")
    import regridding_gb300 as rg
    from regridding_gb300 import workloads

    gi = np.meshgrid(*(np.linspace(-1, 1, n + 1) for n in shape_in), indexing="ij")
    go = workloads.perturb(np.meshgrid(*(np.linspace(-0.9, 0.9, n + 1) for n in shape_out), indexing="ij"))
    ii, oo, vv = rg.build_conservative_2d((gi[0] + 0.1 * gi[1], gi[1] - 0.1 * gi[0]), go).export_numpy()
    order = np.argsort(oo, kind="stable")
    ii, oo, vv = ii[order], oo[order], vv[order]
    n_in, n_out = (int(np.prod(s)) for s in (shape_in, shape_out))
    dw = rg.DeviceWeights.from_coo(ii, oo, vv, n_in, n_out, shape_out, shape_in)
    v = np.random.default_rng(4).lognormal(3, 1, (5, n_in)).astype(np.float32)
    want = np.zeros((5, n_out))
    for d in range(5):
        np.add.at(want[d], oo, vv * v[d, ii].astype(np.float64))
    return torch, dw, torch.from_numpy(v).cuda(), want


def set_shape(dw, which, shape):
    from regridding_gb300 import _lib

    return getattr(_lib.load(), f"rg_weights_set_{which}_shape")(dw.handle, *map(ctypes.c_int64, shape))


def captured(torch, call):
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    return graph


def near(got, want):
    return np.all(np.abs(got.cpu().numpy() - want) <= 1e-12 * want)


@pytest.mark.parametrize("mode", ["exact", "compensated"])
def test_captured_lists_outlive_a_new_shape(mode):
    torch, dw, v, want = handle((41, 43), (30, 33))
    out = torch.empty(want.shape, dtype=torch.float64, device="cuda")
    dw.apply(v, out=out, accumulate=mode)
    graph = captured(torch, lambda: dw.apply(v, out=out, accumulate=mode))
    for which, shape in (("output", (33, 30)), ("input", (43, 41)), ("output", (30, 33))):
        assert set_shape(dw, which, shape) == 0
        assert near(dw.apply(v, accumulate=mode), want)
        spare = torch.full((1 << 20,), 7.0, device="cuda")  # takes memory that the lists would have left
        out.zero_()
        graph.replay()
        assert near(out, want)
        del spare
    dw.free()


def test_applies_beside_new_shapes():
    torch, dw, v, want = handle((41, 43), (30, 33))
    bad = []

    def applies():
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in range(200):
                got = dw.apply(v, accumulate=("exact", "compensated")[k % 2])
                torch.cuda.current_stream().synchronize()
                if not near(got, want):
                    bad.append(k)

    threads = [threading.Thread(target=applies) for _ in range(3)]
    for t in threads:
        t.start()
    k = 0
    while any(t.is_alive() for t in threads) and k < 300:
        assert set_shape(dw, "output", ((33, 30), (30, 33))[k % 2]) == 0
        k += 1
    for t in threads:
        t.join()
    assert not bad
    dw.free()


@pytest.mark.parametrize("calls", ["two float64", "unaligned float32"])
def test_input_shape_stays_open(calls):
    """Calls that stage no aligned float32 rows leave the input shape free."""
    torch, dw, v, want = handle((40, 48), (30, 33))
    if calls == "two float64":
        for _ in range(2):
            dw.apply(v.double())
    else:
        off = torch.empty(v.numel() + 1, device="cuda")[1:].reshape(v.shape)
        off.copy_(v)
        dw.apply(off)
    assert set_shape(dw, "input", (48, 40)) == 0
    for x in (v.double(), v.double(), v):
        np.testing.assert_array_equal(dw.apply(x).cpu().numpy(), want)
    dw.free()


@pytest.mark.parametrize("mode", ["exact", "compensated", "fast"])
def test_input_shape_is_fixed_by_staged_rows(mode):
    from regridding_gb300 import _lib

    torch, dw, v, want = handle((40, 48), (30, 33))
    dw.apply(v, accumulate=mode)
    assert set_shape(dw, "input", (48, 40)) == _lib.RG_ERR_ARG
    assert set_shape(dw, "input", (40, 48)) == 0
    dw.free()


@pytest.mark.parametrize("shape_in", [(41, 43), (40, 48)])
@pytest.mark.parametrize("mode", ["exact", "compensated"])
def test_first_call_under_capture(shape_in, mode):
    """A captured call makes no lists (the host would read them back): where a
    fast apply has made the float32 weights, its gathers are captured."""
    torch, dw, v, want = handle(shape_in, (30, 33))
    out = torch.empty(want.shape, dtype=torch.float64, device="cuda")
    dw.apply(v, accumulate="fast")
    graph = captured(torch, lambda: dw.apply(v, out=out, accumulate=mode))
    for _ in range(2):
        out.zero_()
        graph.replay()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
        assert near(dw.apply(v, accumulate=mode), want)
    dw.free()
