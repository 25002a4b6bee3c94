"""The one-sweep boundary kernels and the Yee sweeps that form their own
boundary ghosts, on the smallest grids, odd ones and both x differences
(se2 = 0: ghosts in the sweeps; se2 != 0: separate boundary sweeps), with
particles up to the faces so that every ghost current is folded.  One
deterministic step is bit-exact against the oracle; the key scan is
exercised below and above its one-launch limit (65536 keys)."""
import numpy as np
import pytest

from aladyn_b200.config import make_params
from aladyn_b200.sim import PicDevice
from oracle.oracle import Oracle
from tests.helpers import grid_small, laser_fields, small_case, sort_records
from tests.test_gpu_tiles import records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("der_ord", [2, 3])
@pytest.mark.parametrize("ndim,nx,ny,nz", [(2, 4, 4, 1), (2, 131, 37, 1), (3, 4, 4, 4), (3, 5, 4, 9), (3, 37, 6, 5)])
def test_boundaries_bitexact(ndim, nx, ny, nz, der_ord):
    out = []
    for cls in (PicDevice, Oracle):
        p = make_params(grid_small(ndim, nx, ny, nz), capacity=(4000, 0, 0, 0), w_sh=0, der_ord=der_ord)
        d = cls(p)
        if cls is PicDevice:
            d.set_deterministic(True)
        d.set_fields(laser_fields(p))
        d.set_species(0, records(p, 2000, "spread", 1.0))
        for it in range(2):
            d.lp_run(it * p.dt, it, initial_time=(it == 0))
        out.append((d.get_fields(), d.get_currents(), d.get_species(0)))
    for a, b in zip(*out):
        assert a.shape == b.shape and np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("nx,ny", [(64, 9), (1000, 250), (2100, 260)])
def test_key_scan_sizes(nx, ny):
    """193, 32769 and 69697 keys: every particle is in the tiles once,
    so the step keeps the count and the particles stay bit-exact."""
    p = small_case(2, nx=nx, ny=ny, cap=60000, w_sh=0)
    rec, ebf = records(p, 50000, "spread", 0.05), laser_fields(p)
    got = []
    for cls in (PicDevice, Oracle):
        d = cls(p)
        d.set_fields(ebf)
        d.set_species(0, rec)
        d.lp_run(0.0, 0, initial_time=True)
        got.append(d.get_species(0))
    assert got[0].shape == got[1].shape
    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))


@pytest.mark.parametrize("der_ord", [2, 3])
@pytest.mark.parametrize("ndim,nx,ny,nz", [(2, 4, 4, 1), (2, 131, 37, 1), (3, 4, 4, 4), (3, 37, 6, 5)])
def test_tiled_steps_with_merged_setup(ndim, nx, ny, nz, der_ord):
    """From the second step on a tiled FP64 species takes the set-up launch
    (field ghosts, cleared currents, histogram) and the particles have only
    to be binned by the step before.  The currents differ from the oracle's by
    the order of their FP64 sums, 1e-12 of the largest value as in
    test_gpu_tiles; three steps multiply that by less than ten."""
    n = 2000
    got = []
    for cls in (PicDevice, Oracle):
        p = make_params(grid_small(ndim, nx, ny, nz), capacity=(n + 16, 0, 0, 0), w_sh=0, der_ord=der_ord)
        d = cls(p)
        d.set_fields(laser_fields(p))
        d.set_species(0, records(p, n, "spread", 1.0))
        for it in range(4):
            d.lp_run(it * p.dt, it, initial_time=(it == 0))
        got.append((d.get_fields(), d.get_currents(), sort_records(d.get_species(0))))
    for a, b in zip(*got):
        assert a.shape == b.shape and np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
