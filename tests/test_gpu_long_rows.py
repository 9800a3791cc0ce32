"""Compensated applies over matrices with long rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape_in,shape_out,lengths,share", [
    ((128, 128), (2, 2), (16000,), 1),            # no box holds a patch
    ((64, 64), (1, 3), (4000,), 1),
    ((56, 60), (48, 48), (3300, 21, 200), 40),    # wide boxes, a few long rows
    ((56, 60), (48, 48), (3300, 21, 200), 2),     # and many
    ((45, 55), (48, 41), (2400, 21, 200), 40),    # rows of any length
    ((45, 55), (48, 41), (2400, 21, 200), 2),
    ((56, 60), (48, 48), (3300, 21, 200), 70),    # few enough to stay
    ((45, 55), (48, 41), (2400, 21, 200), 70),
])
@pytest.mark.parametrize("stack", [1, 3, 64])
@pytest.mark.parametrize("data", ["equal", "lognormal"])
def test_compensated_within_1e_12(shape_in, shape_out, lengths, share, stack, data):
    """Every output of positive data is within 1e-12 of the exact apply's,
    whatever its row's length (rows up to 20 entries by the bound of
    float-float sums of one sign, 9.8e-13); rows too long for that are the exact sums."""
    torch = pytest.importorskip("torch")
    import regridding_gb300 as rg

    rng = np.random.default_rng([3, stack, len(lengths), share])
    n_in, n_out = (int(np.prod(s)) for s in (shape_in, shape_out))
    n = rng.integers(1, 21, n_out)
    long = np.arange(n_out) % share == 0
    n[long] = np.resize(lengths, long.sum())
    ii = np.concatenate([np.sort(rng.choice(n_in, k, replace=False)) for k in n])
    oo = np.repeat(np.arange(n_out), n)
    vv = np.full(ii.size, 1 / 3) if data == "equal" else rng.uniform(0.01, 1, ii.size)
    dw = rg.DeviceWeights.from_coo(ii, oo, vv, n_in, n_out, shape_out, shape_in)
    v = np.full((stack, n_in), 0.1) if data == "equal" else rng.lognormal(3, 1, (stack, n_in))
    v = torch.from_numpy(v.astype(np.float32)).cuda()
    exact = dw.apply(v).cpu().numpy()
    got = dw.apply(v, accumulate="compensated").cpu().numpy()
    np.testing.assert_array_equal(got[:, n > 20], exact[:, n > 20])
    assert np.all(np.abs(got - exact) <= 1e-12 * exact)
    dw.free()
