"""``regrid_from_weights()`` and ``regrid()``.

Host-side structure follows regridding/_regrid/_regrid_from_weights.py:12-162
and regridding/_regrid/_regrid.py:12-149; the apply runs on the GPU
(``rg_apply``), once per distinct weights element over every orthogonal
slice that shares it.
"""

from __future__ import annotations

from typing import Literal, Sequence

import numpy as np

from . import _device, _util
from ._weights import Entries, _weights_device

__all__ = ["regrid_from_weights", "regrid"]


def _shapes(shape_input, shape_output, values_shape, axis_input, axis_output):
    ndim_input = len(shape_input)
    ndim_output = len(shape_output)
    axis_input = _util.normalize_axis(axis_input, ndim=ndim_input)
    axis_output = _util.normalize_axis(axis_output, ndim=ndim_output)
    orth_in = tuple(shape_input[i] for i in _util.normalize_axis(None, ndim_input) if i not in axis_input)
    orth_out = tuple(shape_output[i] for i in _util.normalize_axis(None, ndim_output) if i not in axis_output)
    if values_shape is not None and len(values_shape) > 0:
        orth_val = tuple(values_shape[i] for i in _util.normalize_axis(None, len(values_shape))
                         if i not in axis_input)
    else:
        orth_val = ()
    shape_orth = np.broadcast_shapes(orth_in, orth_out, orth_val)
    axis_input = tuple(sorted(axis_input))
    axis_output = tuple(sorted(axis_output))
    full_in = _util.insert_resampled(shape_orth, tuple(reversed(axis_input)), shape_input)
    full_out = _util.insert_resampled(shape_orth, tuple(reversed(axis_output)), shape_output)
    return axis_input, axis_output, shape_orth, full_in, full_out


def regrid_from_weights(
    weights: np.ndarray,
    shape_input: tuple[int, ...],
    shape_output: tuple[int, ...],
    values_input: np.ndarray,
    values_output: None | np.ndarray = None,
    axis_input: None | int | Sequence[int] = None,
    axis_output: None | int | Sequence[int] = None,
    *,
    accumulate: Literal["exact", "fast", "compensated"] = "exact",
) -> np.ndarray:
    """Apply saved weights to an array (drop-in for ``regridding.regrid_from_weights``).

    The default ``accumulate="exact"`` gives the upstream float64 result bit
    for bit (or, for a float32 ``values_output``, the upstream in-place
    float32 result).  ``accumulate="fast"`` accumulates in the output dtype
    with FMA (float32 output for float32 input unless ``values_output`` says
    otherwise): the HBM-bandwidth path, within about 1e-6 relative of the
    float64 result.  ``accumulate="compensated"`` returns the upstream's
    float64 output within 1e-12 relative of it where a sum's terms have one
    sign, computed for float32 input in float-float arithmetic on the FP32
    pipe (long rows in float64), about 5x faster than ``"exact"`` on GB300
    (other inputs compute as ``"exact"``).
    """
    return _apply(weights, shape_input, shape_output, values_input, values_output, axis_input, axis_output, accumulate)


def _apply(weights, shape_input, shape_output, values_input, values_output, axis_input, axis_output, accumulate):
    """:func:`regrid_from_weights`; ``weights`` may also be the 1D
    :class:`Entries` of a build that never left the device."""
    if accumulate not in ("exact", "fast", "compensated"):
        raise ValueError(f"accumulate must be 'exact', 'fast' or 'compensated', got {accumulate!r}")
    unit = getattr(values_input, "unit", None)
    if unit is not None:
        values_input = getattr(values_input, "value")
    values_input = np.asarray(values_input)

    axis_input, axis_output, shape_orth, full_in, full_out = _shapes(
        shape_input, shape_output, values_input.shape if np.ndim(values_input) > 0 else (), axis_input,
        axis_output)

    entries = element = None
    if isinstance(weights, Entries):
        n_cells = [int(np.prod([shape[ax] for ax in axes])) for shape, axes in
                   ((full_in, axis_input), (full_out, axis_output))]
        if weights.ind_in.shape[0] == 1:
            one = np.empty(weights.shape, dtype=object)
            one[...] = _DeviceElement(_device.DeviceWeights.block_diagonal(
                weights.ind_in, weights.ind_out, weights.val, weights.count, *n_cells))
            weights = one
        else:
            entries = weights
            element = np.arange(entries.ind_in.shape[0]).reshape(entries.shape)
            element = np.broadcast_to(element, shape_orth).reshape(-1)
            weights = np.empty(0, dtype=object)
    w_arr = weights if entries is not None else np.broadcast_to(np.array(weights), shape_orth, subok=True)
    values_input = np.broadcast_to(values_input, full_in, subok=True)

    out_dtype = np.float64
    if values_output is None:
        if accumulate == "fast" and values_input.dtype == np.float32:
            out_dtype = np.float32
        # every element is written below; pages pre-faulted for the copy-back
        values_output = _device.host_empty(full_out, out_dtype)
    else:
        if values_output.shape != full_out:
            raise ValueError(f"{values_output.shape=} should be equal to {full_out}")
        values_output.fill(0)

    numba_in = _util.numba_axes(len(axis_input))
    numba_out = _util.numba_axes(len(axis_output))
    shape_in_numba = tuple(full_in[ax] for ax in axis_input)
    shape_out_numba = tuple(full_out[ax] for ax in axis_output)
    n_in = int(np.prod(shape_in_numba))
    n_out = int(np.prod(shape_out_numba))

    v_in = np.moveaxis(values_input, axis_input, numba_in).reshape(-1, n_in)
    v_out_view = np.moveaxis(values_output, axis_output, numba_out)
    shape_out_tmp = v_out_view.shape

    flat = w_arr.reshape(-1)
    unit_weights = getattr(flat[0][2], "unit", None) if flat.size and not isinstance(
        flat[0], _DeviceElement) else None

    t = _device.torch()
    in_dtype = values_input.dtype
    if in_dtype not in (np.float32, np.float64):
        in_dtype = np.float64
    out_np_dtype = values_output.dtype if values_output.dtype in (np.float32, np.float64) else np.float64

    # group the orthogonal slices by the weights element they use
    groups: dict[int, list[int]] = {}
    first: dict[int, int] = {}
    for d in range(flat.size):
        key = id(flat[d])
        if key not in groups:
            groups[key] = []
            first[key] = d
        groups[key].append(d)

    if entries is None and len(axis_input) == 1:
        entries, element = _short_elements(flat, groups, first)
    if entries is not None:
        groups = {}

    # one matrix and a row-major output view: the device result is copied
    # straight into values_output
    direct = None
    if (len(groups) == 1 or entries is not None) and v_out_view.flags.c_contiguous and \
            v_out_view.dtype == out_np_dtype:
        direct = v_out_view.reshape(v_in.shape[0], n_out)
    result = None if direct is not None else np.empty((v_in.shape[0], n_out), dtype=out_np_dtype)
    if entries is not None:
        _apply_blocks(entries, n_in, n_out, element, v_in, in_dtype, result if direct is None else direct, accumulate)
    d_all = None
    if len(groups) == 1:
        d_all = _device.upload(v_in, in_dtype)
    for key, rows in groups.items():
        element = flat[first[key]]
        if isinstance(element, _DeviceElement):
            dw = element.dw
        else:
            dw = _device.lookup(element, n_in, n_out)
        if dw is None:
            ii, oo, vv = element
            vv = getattr(vv, "value", vv)
            dw = _device.DeviceWeights.from_coo(np.asarray(ii), np.asarray(oo), np.asarray(vv, dtype=np.float64),
                                                n_in, n_out, shape_out_numba, shape_in_numba)
            _device.remember(element, dw)
        if d_all is not None:
            src = d_all
        else:
            src = _device.upload(v_in[rows], in_dtype)
        dst = t.empty((len(rows), n_out), dtype=_device.torch_dtype(out_np_dtype), device="cuda")
        dw.apply(src, out=dst, accumulate=accumulate)
        if direct is not None:
            t.from_numpy(direct).copy_(dst)
        elif d_all is not None and len(rows) == flat.size:
            result[:] = _device.download(dst)
        else:
            result[rows] = _device.download(dst)

    if result is not None:
        v_out_view[...] = result.reshape(shape_out_tmp)
    values_output = np.moveaxis(v_out_view, numba_out, axis_output)

    if unit_weights is not None:
        unit = unit_weights if unit is None else unit * unit_weights
    if unit is None:
        return values_output
    return values_output << unit


# Saved 1D elements of up to this many entries on average are applied as one
# block diagonal matrix, uploaded on each call: an element of its own takes
# about 0.2 ms (with its device copy kept) to 0.45 ms of launches and copies,
# and the upload of 16384 entries about 0.1 ms.
SHORT_ELEMENT = 16384


def _short_elements(flat: np.ndarray, groups: dict, first: dict):
    """The short saved elements of ``groups`` as device :class:`Entries` and
    the element of every flat slice, or ``(None, None)`` where they are long
    or few or not used by equally many slices."""
    if len(groups) < 4 or len({len(rows) for rows in groups.values()}) > 1:
        return None, None
    elements = [flat[first[key]] for key in groups]
    if any(isinstance(e, _DeviceElement) for e in elements):
        return None, None
    arrays = [(np.asarray(ii), np.asarray(oo), np.asarray(getattr(vv, "value", vv), dtype=np.float64))
              for ii, oo, vv in elements]
    count = np.array([vv.size for *_, vv in arrays], dtype=np.int64)
    stride = int(count.max())
    if stride * len(arrays) > 2 * int(count.sum()) or count.mean() > SHORT_ELEMENT or any(
            a.ndim != 1 or a.size != c for e, c in zip(arrays, count) for a in e):
        return None, None
    element = np.empty(flat.size, dtype=np.int64)
    for k, rows in enumerate(groups.values()):
        element[rows] = k
    host = [np.zeros((len(arrays), stride), dtype=dtype) for dtype in (np.int64, np.int64, np.float64)]
    for k, e in enumerate(arrays):
        for h, a in zip(host, e):
            h[k, :a.size] = a
    return Entries(*(_device.upload(h) for h in host), _device.upload(count), (len(arrays),)), element


# Input and output of a block diagonal matrix's slices on the device, at most
# (an element's own slices are never cut).
BLOCK_BYTES = 1 << 30


def _apply_blocks(entries, n_in: int, n_out: int, element: np.ndarray, v_in: np.ndarray, in_dtype, out: np.ndarray,
                  accumulate: str) -> None:
    """Slice ``d`` of ``v_in`` through element ``element[d]`` of the device
    ``entries`` into ``out[d]``: block diagonal matrices over as many
    elements as 2^31 cells and BLOCK_BYTES hold, each with one apply.  (The
    elements one by one, 256 spectra of 512 -> 384 cells: 118 ms.)"""
    t = _device.torch()
    if element.size == 0:
        return
    nd, stride = entries.ind_in.shape
    nbytes = element.size // nd * (n_in * np.dtype(in_dtype).itemsize + n_out * out.dtype.itemsize)
    most = max(1, min((2**31 - 2) // max(n_in, n_out, 1), (2**32 - 2) // max(stride, 1), BLOCK_BYTES // max(nbytes, 1)))
    # slices of an element side by side: (slices, elements)
    order = np.argsort(element, kind="stable").reshape(nd, -1)
    for d in range(0, nd, most):
        rows = order[d:d + most].T
        count = None if entries.count is None else entries.count[d:d + most]
        dw = _device.DeviceWeights.block_diagonal(entries.ind_in[d:d + most], entries.ind_out[d:d + most],
                                                  entries.val[d:d + most], count, n_in, n_out)
        at = rows.reshape(-1)
        if np.array_equal(at, np.arange(at[0], at[0] + at.size)):
            at = slice(at[0], at[0] + at.size)
        src = _device.upload(v_in[at], in_dtype)
        dst = t.empty((rows.shape[0], rows.shape[1] * n_out), dtype=_device.torch_dtype(out.dtype), device="cuda")
        dw.apply(src.reshape(rows.shape[0], -1), out=dst, accumulate=accumulate)
        if isinstance(at, slice):
            t.from_numpy(out[at]).copy_(dst.reshape(-1, n_out))
        else:
            out[at] = _device.download(dst).reshape(-1, n_out)
        dw.free()


class _DeviceElement:
    """Stand-in for a saved-layout element whose weights live only on the GPU."""

    __slots__ = ("dw",)

    def __init__(self, dw):
        self.dw = dw

    def __getitem__(self, k):
        return None


def regrid(
    coordinates_input: tuple[np.ndarray, ...],
    coordinates_output: tuple[np.ndarray, ...],
    values_input: np.ndarray,
    values_output: None | np.ndarray = None,
    axis_input: None | int | Sequence[int] = None,
    axis_output: None | int | Sequence[int] = None,
    method: Literal["multilinear", "conservative"] = "multilinear",
    bounds: Literal["extrapolate", "nan", "raise"] = "extrapolate",
    perturb: None | bool = None,
    seed: "None | int | np.random.Generator" = _util.SEED_DEFAULT,
    *,
    accumulate: Literal["exact", "fast", "compensated"] = "exact",
) -> np.ndarray:
    """Regrid in one call (drop-in for ``regridding.regrid``).

    Builds the weights on the GPU and applies them without a round trip of
    the weights through host memory; the result is bit-identical to
    ``regrid_from_weights(*weights(...), ...)``.
    """
    array, shape_in, shape_out, dev = _weights_device(
        coordinates_input, coordinates_output, axis_input, axis_output, None, method, bounds, perturb, seed,
        want_host=False)
    if isinstance(dev, Entries):
        return _apply(dev, shape_in, shape_out, values_input, values_output, axis_input, axis_output, accumulate)
    if array is None:
        # 2D conservative: one device matrix per orthogonal element
        *_, shape_orth = _util.normalize_input_output_coordinates(
            coordinates_input, coordinates_output, axis_input, axis_output)
        array = np.empty(len(dev), dtype=object)
        for k, dw in enumerate(dev):
            array[k] = _DeviceElement(dw)
        array = array.reshape(shape_orth)
    return regrid_from_weights(array, shape_in, shape_out, values_input, values_output, axis_input,
                               axis_output, accumulate=accumulate)
