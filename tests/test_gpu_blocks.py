"""Stacks over many 1D elements, applied block by block."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["elements first", "stack first"])
def test_device_stacks_stay_bounded(monkeypatch, order):
    """1.6 GB of float32 slices over eight elements: no upload takes more
    than 1 GiB, and every slice is its element's exact sum."""
    pytest.importorskip("torch")
    import regridding_gb300 as rg
    from regridding_gb300 import _device

    rng = np.random.default_rng(8)
    nd, slices, n, m = 8, 50_000, 1000, 40
    x = np.sort(rng.uniform(0, 1, (nd, n + 1)), axis=1)
    y = np.linspace(0.1, 0.9, m + 1)
    v = rng.integers(0, 100, n).astype(np.float32)
    shape = (nd, slices, n) if order == "elements first" else (slices, nd, n)
    values = np.broadcast_to(v, shape)
    if order == "elements first":
        x = x[:, None]
    sizes = []
    upload = _device.upload

    def counted(a, *args, **kwargs):
        sizes.append(a.nbytes)
        return upload(a, *args, **kwargs)

    monkeypatch.setattr(_device, "upload", counted)
    out = rg.regrid((x,), (y,), values, axis_input=-1, axis_output=-1, method="conservative", accumulate="fast")
    assert max(sizes) <= 1 << 30
    assert out.shape == shape[:-1] + (m,)
    one = rg.regrid((x,), (y,), np.broadcast_to(v, shape[:2] + (n,))[:1, :1] if nd == 1 else
                    (values[:, :1] if order == "elements first" else values[:1]),
                    axis_input=-1, axis_output=-1, method="conservative", accumulate="fast")
    assert np.array_equal(out, np.broadcast_to(one, out.shape))
