"""Failure paths of the build, exercised on the GPU without a GPU fault.

* An undersized triple buffer: RG_FAULT_CHUNK_SLOTS caps the slots each
  chunk of the parallel walk gets, so chunks overflow their buffers (the
  device flags it; nothing is written past a buffer) and the build takes its
  recovery path, whole-line walks sized by an exact count.  The weights are
  bit-identical to the normal build's and to the oracle's.
* The debug library (RG_DEBUG=1: bounds-checked grid reads in the builds,
  an out-of-range read recorded as an error status rather than a trap)
  builds, loads, and gives the release library's weights bit for bit.
"""

import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from test_gpu_parity import assert_same, distorted, rect

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rg():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import regridding_gb300

    return regridding_gb300


def test_undersized_chunk_slots_take_the_recovery_path(rg, monkeypatch):
    from regridding_gb300 import _device, workloads

    gi = distorted(257, 0.25, 0.02)
    go = workloads.perturb(rect(193, -1.05, 1.05))
    ref = rg.build_conservative_2d(gi, go).export_numpy()
    monkeypatch.setenv("RG_FAULT_CHUNK_SLOTS", "4")
    got = rg.build_conservative_2d(gi, go).export_numpy()
    for g, r, e in zip(got, ref, oracle.weights_conservative_2d(gi, go)):
        assert_same(g, r)
        assert_same(g, e)
    # batched builds take the same path for the whole batch
    rng = np.random.default_rng(12)
    pairs = [workloads.grid_pair(rng, side) for side in (40, 97, 150)]
    batched = _device.build_conservative_2d_batch(pairs)
    for (pgi, pgo), dw in zip(pairs, batched):
        for g, e in zip(dw.export_numpy(), oracle.weights_conservative_2d(pgi, pgo)):
            assert_same(g, e)


def test_graded_grids_keep_to_their_chunks(rg):
    """Lines that lie ten times as far apart at the rim as in the middle fit
    the chunks' slots: a build takes about twice that of even lines (by whole
    lines, after an overflow, twelve times)."""
    import time

    import torch

    from regridding_gb300 import workloads

    x, y = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in workloads.distorted_grid(513, 0.1, 0.02))
    even = workloads.perturb(workloads.rect_grid(385, -0.95, 0.95))
    seconds = []
    for power in (1, 2):
        go = [torch.from_numpy(np.sign(a) * np.abs(a) ** power).cuda() for a in even]
        times = []
        for _ in range(6):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            dw = rg.build_conservative_2d((x, y), go)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
            dw.free()
        seconds.append(min(times))
    assert seconds[1] < 5 * seconds[0], seconds


def test_cycling_walks_end_soon(rg, monkeypatch):
    """A pair whose walk cycles around a shared vertex is reported about as
    soon as its whole lines are walked: the line's further chunks are not
    walked to their step caps, too (five times as long)."""
    import time

    import torch

    from regridding_gb300 import workloads

    gi, go = ([torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in g]
              for g in (workloads.distorted_grid(65, 0.3, 0.02), workloads.rect_grid(49, -1.05, 1.05)))
    seconds = []
    for chunk in ("0", None):
        monkeypatch.setenv("RG_SWEEP_CHUNK", chunk) if chunk else monkeypatch.delenv("RG_SWEEP_CHUNK")
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        with pytest.raises(rg.RegridError, match="step cap"):
            rg.build_conservative_2d(gi, go)
        seconds.append(time.perf_counter() - t0)
    assert seconds[1] < 3 * seconds[0], seconds


def test_debug_library_builds_and_matches():
    code = f"""
import sys
sys.path.insert(0, {ROOT!r})
sys.path.insert(0, {os.path.join(ROOT, 'tests')!r})
import numpy as np
import oracle
import regridding_gb300 as rg
from regridding_gb300 import _lib, workloads
assert _lib.library_path().endswith('_build_debug/libregrid_gb300.so'), _lib.library_path()
gi = workloads.distorted_grid(129, 0.3, 0.02)
go = workloads.perturb(workloads.rect_grid(97, -1.05, 1.05))
got = rg.build_conservative_2d(gi, go).export_numpy()
for g, e in zip(got, oracle.weights_conservative_2d(gi, go)):
    assert np.array_equal(g, e)
print('debug ok', _lib.load()._name)
"""
    env = dict(os.environ, RG_DEBUG="1")
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=900)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "debug ok" in res.stdout


def test_debug_library_reports_a_single_pairs_bounds():
    """A bounds word set while one pair is built (here by the host, as a read
    outside an array would) fails that build, and not the next one."""
    code = f"""
import sys
sys.path.insert(0, {ROOT!r})
import regridding_gb300 as rg
from regridding_gb300 import _lib, workloads
gi = workloads.distorted_grid(33, 0.3, 0.02)
go = workloads.perturb(workloads.rect_grid(25, -1.05, 1.05))
rg.build_conservative_2d(gi, go)
assert _lib.load().rg_debug_out_of_bounds() == _lib.RG_OK
try:
    rg.build_conservative_2d(gi, go)
except rg.RegridError as e:
    assert 'bounds check' in str(e), e
else:
    raise SystemExit('not reported')
rg.build_conservative_2d(gi, go)
print('reported')
"""
    env = dict(os.environ, RG_DEBUG="1")
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=900)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "reported" in res.stdout
