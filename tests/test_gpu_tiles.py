"""The tiled particle kernels where their paths meet: rows that end inside a
group or fill several, nodes with more particles than a node's list holds,
particles that change node (many, few, all), grids whose last tiles are
partial, box edges.  One step against the oracle.

Tolerance of the FP64 currents: a node sums at most a few thousand terms of
either sign in another order, each rounded to 2^-53 of at most the largest
|J|: 1e-12 of the largest |J|; particles are bit-exact.
"""
import numpy as np
import pytest

from aladyn_b200.abi import AGPU_FP64
from aladyn_b200.sim import PicDevice, pack_slot
from oracle.oracle import Oracle
from tests.helpers import laser_fields, small_case

pytestmark = pytest.mark.gpu

# grid and records: spread over the box, or piled up in a few cells
CASES = [(2, 31, 7, 1, 700, "spread"), (2, 64, 9, 1, 3000, "piled"), (2, 97, 23, 1, 20000, "spread"),
         (3, 31, 5, 4, 900, "spread"), (3, 33, 6, 7, 4000, "piled"), (3, 70, 13, 9, 30000, "spread")]


def records(p, n, how, pmax, seed=3):
    r = np.random.default_rng(seed)
    nd = p.ndim
    lo, hi = [p.gxmin, p.gymin, p.gzmin][:nd], [p.gxmax, p.gymax, p.gzmax][:nd]
    rec = np.zeros((n, 2 * nd + 1), order="F")
    for a in range(nd):
        u = r.random(n)
        if how == "piled":  # half of the records in one cell, the rest in a few
            u = np.where(r.random(n) < 0.5, 0.4 + 0.002 * u, 0.35 + 0.15 * u)
        rec[:, a] = lo[a] + (hi[a] - lo[a]) * (1e-9 + (1 - 2e-9) * u)
        rec[:, nd + a] = pmax * (2 * r.random(n) - 1)
    rec[:, 2 * nd] = pack_slot(np.full(n, -1), np.zeros(n), r.random(n).astype(np.float32) + 0.5)
    return rec


def step(cls, p, rec, ebf):
    d = cls(p)
    d.set_fields(ebf)
    d.set_species(0, rec)
    d.lp_run(0.0, 0, initial_time=True)
    return d


@pytest.mark.parametrize("pmax", [0.0, 0.05, 5.0])
@pytest.mark.parametrize("ndim,nx,ny,nz,n,how", CASES)
def test_fp64_tile_step(ndim, nx, ny, nz, n, how, pmax):
    p = small_case(ndim, nx=nx, ny=ny, nz=nz, cap=n + 16, precision=AGPU_FP64)
    rec, ebf = records(p, n, how, pmax), laser_fields(p)
    dev, ora = step(PicDevice, p, rec, ebf), step(Oracle, p, rec, ebf)
    a, b = dev.get_species(0), ora.get_species(0)
    assert a.shape == b.shape
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
    ja, jb = dev.get_currents(), ora.get_currents()
    assert np.abs(ja - jb).max() <= 1e-12 * np.abs(jb).max()

