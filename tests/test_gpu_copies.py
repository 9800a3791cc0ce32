"""Host bytes to the device: with the launch, by a kernel, and the sizes where
one gives way to the next."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 3967, 3968, 3969, 31999, 32000, 32001, 64000, 95999, 96000, 96001, 300003])
@pytest.mark.parametrize("shift", [0, 1, 4, 8])
def test_copy_from_host(n, shift):
    torch = pytest.importorskip("torch")
    from regridding_gb300 import _device, _lib

    a = np.random.default_rng(n).integers(0, 256, n + shift, dtype=np.uint8)
    d = torch.full((n + shift + 64,), 7, dtype=torch.uint8, device="cuda")
    _lib.call("rg_copy_from_host", ctypes.c_void_p(d.data_ptr() + shift), ctypes.c_void_p(a.ctypes.data + shift), n,
              _device.stream())
    want = a[shift:].copy()
    a[:] = 0  # the source has been read
    got = d.cpu().numpy()
    np.testing.assert_array_equal(got[shift:shift + n], want)
    assert np.all(got[:shift] == 7) and np.all(got[shift + n:] == 7)
