"""The counts a host reads: particles alive, pushed and removed, in the
synchronous steps, with deferred counts and with replayed step graphs.
Particles are bit-exact in the first FP64 step and to rounding after it, so
counts are compared exactly."""
import os
import subprocess
import sys

import numpy as np
import pytest

from aladyn_b200.abi import AGPU_FP32_SPLIT, AGPU_FP64
from aladyn_b200.sim import PicDevice
from oracle.oracle import Oracle
from tests.helpers import laser_fields, small_case, sort_records
from tests.test_gpu_tiles import records

pytestmark = pytest.mark.gpu


def _dev(cls, p, rec):
    d = cls(p)
    d.set_fields(laser_fields(p))
    for ic in range(p.nsp_run):
        d.set_species(ic, rec[ic::p.nsp_run])
    return d


def _step(d, p, it):
    out = d.lp_run(it * p.dt, it, initial_time=(it == 0))
    return out[1] if isinstance(out, tuple) else out


@pytest.mark.parametrize("graphs", [False, True])
def test_deferred_counts_between_steps(graphs):
    """Diagnostics after every step while particles leave the box: the count,
    the sums and the pushes are those of synchronous steps, whether a step is
    launched, captured or replayed."""
    p = small_case(2, cap=30000, w_sh=0)
    rec = records(p, 20000, "spread", 5.0)
    a, b = _dev(PicDevice, p, rec), _dev(PicDevice, p, rec)
    b.set_deferred_counts(True)
    b.set_step_graphs(graphs)
    last = 20000
    for it in range(8):
        oa = _step(a, p, it)
        _step(b, p, it)
        da, db = a.diag(), b.diag()
        assert oa.np[0] == da.np[0] < last
        last = da.np[0]
        assert db.np[0] == da.np[0], it
        assert abs(db.kin_energy[0] - da.kin_energy[0]) <= 1e-9 * da.kin_energy[0]
    assert b.timers().pushes == a.timers().pushes
    assert b.get_species(0).shape == a.get_species(0).shape


def test_tiles_after_a_deterministic_step():
    """A deterministic step moves the particles without new binning keys: the
    tiled step after it bins them again."""
    p = small_case(2, cap=30000, w_sh=0)
    rec = records(p, 20000, "piled", 1.0)  # away from the faces: nothing is removed
    dev, ora = _dev(PicDevice, p, rec), _dev(Oracle, p, rec)
    for it in range(4):
        dev.set_deterministic(it == 1)
        out, oo = _step(dev, p, it), _step(ora, p, it)
        assert out.error_bits == 0 and out.np[0] == oo.np[0] == 20000, it
    a, b = sort_records(dev.get_species(0)), sort_records(ora.get_species(0))
    assert np.abs(a[:, :4] - b[:, :4]).max() <= 1e-12 * np.abs(b[:, :4]).max()


@pytest.mark.parametrize("precision", [AGPU_FP64, AGPU_FP32_SPLIT])
def test_removed_counts_over_window_steps(precision):
    """agpu_step_out.removed holds this step's drops, on window steps too:
    np = np before - removed + injected, and the oracle's number (FP64)."""
    p = small_case(2, cap=30000, w_sh=3, precision=precision)
    rec = records(p, 20000, "spread", 5.0)
    dev, ora = _dev(PicDevice, p, rec), _dev(Oracle, p, rec)
    last, shifts = 20000, 0
    for it in range(10):
        out, oo = _step(dev, p, it), _step(ora, p, it)
        assert out.np[0] == last - out.removed[0] + out.injected[0], it
        if precision == AGPU_FP64:
            assert out.removed[0] == oo.removed[0] > 0 and out.np[0] == oo.np[0], it
        last, shifts = out.np[0], shifts + (out.nshx > 0)
    assert shifts >= 2


# cudaMemcpyAsync with one device-to-host copy that fails on the host, when armed
SHIM = """
#include <dlfcn.h>
#include <stddef.h>
int armed = 0;
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) {
  static int (*real)(void*, const void*, size_t, int, void*);
  if (!real) real = (int (*)(void*, const void*, size_t, int, void*))dlsym(
      dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaMemcpyAsync");
  if (armed && kind == 2) { armed = 0; return 2; }
  return real(d, s, n, kind, st);
}
"""
FAILED_READ = """
import ctypes, sys
from aladyn_b200.sim import PicDevice
from tests.helpers import small_case
from tests.test_gpu_counts import _dev, _step
from tests.test_gpu_tiles import records
armed = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "armed")
p = small_case(2, cap=30000, w_sh=0)
rec = records(p, 20000, "spread", 5.0)
a, b = _dev(PicDevice, p, rec), _dev(PicDevice, p, rec)
for it in range(4):
    n = _step(a, p, it).np[0]
    armed.value = it == 1
    try:
        _step(b, p, it)
        assert it != 1
    except RuntimeError:
        assert it == 1 and armed.value == 0
        assert b.count(0) == n < 20000, (b.count(0), n)
        assert b.diag().np[0] == n
assert b.count(0) == a.count(0) and b.get_species(0).shape == a.get_species(0).shape
print("counts ok")
"""


def test_counts_after_a_failed_read(tmp_path):
    """A step whose read of the counts fails (a host-side fake of the copy)
    returns an error; the counts are read at the next call."""
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FAILED_READ, str(lib)], cwd=root, capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(lib)), timeout=300)
    assert r.returncode == 0 and "counts ok" in r.stdout, r.stdout + r.stderr
