"""The patch kernel's wide boxes on the GPU against the sums in numpy."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape_in,shape_out,angle", [
    ((40, 40), (30, 30), 0.1),      # one 32-column box would do, rows of 160 bytes
    ((41, 43), (30, 33), 0.1),      # rows of any length
    ((96, 96), (72, 72), 0.5),      # footprints over 32 columns
    ((97, 95), (72, 71), 0.5),
    ((96, 100), (40, 42), 0.4),     # coarse output cells, long rows
    ((300, 24), (225, 18), 0.5),    # input cells of unequal sides: patches of 64 x 4
    ((24, 300), (18, 225), 0.5),    # and of 4 x 64
    ((128, 128), (24, 24), 0.3),    # no box holds a patch
    ((3, 5), (2, 3), 0.1),
    ((1, 7), (1, 5), 0.0),
])
@pytest.mark.parametrize("stack", [1, 2, 3, 4, 9])
def test_wide_boxes_match_plain_apply(shape_in, shape_out, angle, stack):
    """Applies of float32 stacks over grids whose patches need wide boxes or
    have unaligned rows: exact bit for bit, compensated within its stated
    bound, fast within float32 chains' (n + 1) 2^-24 sum |w x|; also from a
    buffer off a 16-byte boundary and with values that are not finite."""
    torch = pytest.importorskip("torch")
    import regridding_gb300 as rg
    from regridding_gb300 import workloads

    rng = np.random.default_rng(5)
    gi = np.meshgrid(*(np.linspace(-1, 1, n + 1) for n in shape_in), indexing="ij")
    c, s = np.cos(angle), np.sin(angle)
    gi = c * gi[0] - s * gi[1], s * gi[0] + c * gi[1]
    go = workloads.perturb(np.meshgrid(*(np.linspace(-0.95, 0.97, n + 1) for n in shape_out), indexing="ij"))
    dw = rg.build_conservative_2d(gi, go)
    ii, oo, vv = dw.export_numpy()
    order = np.argsort(oo, kind="stable")
    ii, oo, vv = ii[order], oo[order], vv[order]
    buffer = torch.from_numpy(rng.lognormal(3, 1, stack * dw.n_in + 1).astype(np.float32)).cuda()
    longest = np.bincount(oo, minlength=dw.n_out).max()
    for offset, special in ((0, False), (1, False), (0, True)):
        v = buffer[offset:offset + stack * dw.n_in].reshape(stack, -1).clone() if offset == 0 else \
            buffer[offset:offset + stack * dw.n_in].reshape(stack, -1)
        if special:
            v[0, dw.n_in // 2], v[-1, 0], v[0, -1] = float("nan"), float("inf"), -3e38
        x = v.cpu().numpy().astype(np.float64)
        want = np.zeros((stack, dw.n_out))
        size = np.zeros((stack, dw.n_out))
        for d in range(stack):
            np.add.at(want[d], oo, vv * x[d, ii])
            np.add.at(size[d], oo, np.abs(vv * x[d, ii]))
        got = dw.apply(v, accumulate="exact").cpu().numpy()
        np.testing.assert_array_equal(got, want)
        for mode, eps in (("compensated", 1.1e-14 + (longest + 2) ** 2 * 3.6e-15), ("fast", (longest + 1) * 2.0 ** -24)):
            got = dw.apply(v, accumulate=mode).cpu().numpy().astype(np.float64)
            fine = np.isfinite(want) & (size < 1e38)
            assert np.array_equal(np.isnan(got), np.isnan(want)) or mode == "fast"
            assert np.all(np.abs(got - want)[fine] <= (eps * size)[fine] + 1e-300), (mode, offset, special)
    dw.free()


@pytest.mark.parametrize("shape_in,shape_out,angle", [
    ((64, 64), (48, 48), 0.05),     # swizzled boxes for float32, wide ones here
    ((32, 32), (24, 24), 0.05),     # the narrowest of those
    ((41, 43), (30, 33), 0.1), ((96, 96), (72, 72), 0.5), ((97, 95), (72, 71), 0.5), ((96, 100), (40, 42), 0.4),
    ((300, 24), (225, 18), 0.5), ((128, 128), (24, 24), 0.3), ((3, 5), (2, 3), 0.1),
])
@pytest.mark.parametrize("stack", [1, 2, 3, 5])
def test_float64_stacks_keep_their_bits(shape_in, shape_out, angle, stack):
    """Exact applies of float64 stacks: the first gathers, later ones stage
    boxes; every one gives the sums in stored order, also when captured, from
    a buffer off a 16-byte boundary, and with values that are not finite."""
    torch = pytest.importorskip("torch")
    import regridding_gb300 as rg
    from regridding_gb300 import workloads

    rng = np.random.default_rng(6)
    gi = np.meshgrid(*(np.linspace(-1, 1, n + 1) for n in shape_in), indexing="ij")
    c, s = np.cos(angle), np.sin(angle)
    gi = c * gi[0] - s * gi[1], s * gi[0] + c * gi[1]
    go = workloads.perturb(np.meshgrid(*(np.linspace(-0.95, 0.97, n + 1) for n in shape_out), indexing="ij"))
    dw = rg.build_conservative_2d(gi, go)
    ii, oo, vv = dw.export_numpy()
    order = np.argsort(oo, kind="stable")
    ii, oo, vv = ii[order], oo[order], vv[order]
    buffer = torch.from_numpy(rng.lognormal(3, 1, stack * dw.n_in + 1)).cuda()
    buffer[5 % dw.n_in] = float("nan")
    buffer[dw.n_in // 2] = float("inf")

    def check(v, got):
        x = v.cpu().numpy()
        want = np.zeros((stack, dw.n_out))
        for d in range(stack):
            np.add.at(want[d], oo, vv * x[d, ii])
        np.testing.assert_array_equal(got.cpu().numpy(), want)

    for offset, mode in ((0, "exact"), (0, "exact"), (0, "compensated"), (1, "exact"), (0, "exact")):
        v = buffer[offset:offset + stack * dw.n_in].reshape(stack, -1)
        check(v, dw.apply(v, accumulate=mode))
    v, out = buffer[:-1].reshape(stack, -1), torch.empty(stack, dw.n_out, dtype=torch.float64, device="cuda")
    fresh = rg.DeviceWeights.from_coo(ii, oo, vv, dw.n_in, dw.n_out, shape_out, shape_in)
    fresh.apply(v, out=out)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        fresh.apply(v, out=out)
    out.zero_()
    graph.replay()
    check(v, out)
