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

from aladyn_b200.abi import AGPU_EBIT_INDEX, AGPU_FP32_SPLIT, AGPU_FP64
from aladyn_b200.sim import PicDevice, pack_slot
from oracle.oracle import Oracle
from tests.helpers import laser_fields, small_case, sort_records

pytestmark = pytest.mark.gpu

# grid and records: spread over the box, or piled up in a few cells
CASES = [(2, 31, 7, 1, 700, "spread"), (2, 64, 9, 1, 3000, "piled"), (2, 97, 23, 1, 20000, "spread"),
         (3, 31, 5, 4, 900, "spread"), (3, 33, 6, 7, 4000, "piled"), (3, 70, 13, 9, 30000, "spread")]


# every node's octants filled alike: the regular tiles of the split form's
# one-node-per-thread path, and the last, partial ones
LATTICE = (3, 66, 9, 9, 8 * 66 * 9 * 9, "lattice")


def records(p, n, how, pmax, seed=3):
    r = np.random.default_rng(seed)
    nd = p.ndim
    lo, hi = [p.gxmin, p.gymin, p.gzmin][:nd], [p.gxmax, p.gymax, p.gzmax][:nd]
    rec = np.zeros((n, 2 * nd + 1), order="F")
    for a in range(nd):
        u = r.random(n)
        if how == "lattice":
            cells = [p.nx, p.ny, p.nz]
            q = np.arange(n) // int(np.prod([2 * c for c in cells[:a]], dtype=np.int64)) % (2 * cells[a])
            u = (q + 0.4 + 0.2 * u) / (2 * cells[a])
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


@pytest.mark.parametrize("pmax", [0.05, 5.0])
@pytest.mark.parametrize("ndim,nx,ny,nz,n,how", CASES + [LATTICE])
def test_split_tile_step(ndim, nx, ny, nz, n, how, pmax):
    """The split form.  A record's offsets are rounded to
    2^-25 cells and each current term to a few times 2^-24 of q w, so against
    displacements of 0.02 cells and more (pmax = 0.05) the currents are off by
    less than 1e-4 of their norm; positions by 2^-24 of a cell, momenta by a
    few 2^-24 of the largest one."""
    got = []
    for cls, prec in ((PicDevice, AGPU_FP32_SPLIT), (Oracle, AGPU_FP64)):
        p = small_case(ndim, nx=nx, ny=ny, nz=nz, cap=n + 16, precision=prec)
        d = step(cls, p, records(p, n, how, pmax), laser_fields(p))
        got.append((d.get_species(0), d.get_currents()))
    (a, ja), (b, jb) = got
    assert a.shape == b.shape
    cell = [p.dx, p.dy, p.dz]
    for c in range(ndim):
        assert np.abs(a[:, c] - b[:, c]).max() <= 4e-7 * cell[c]
        assert np.abs(a[:, ndim + c] - b[:, ndim + c]).max() <= 4e-6 * np.abs(b[:, ndim:2 * ndim]).max()
    assert np.linalg.norm(ja - jb) <= 1e-4 * np.linalg.norm(jb)


def env_step(cls, p, ep, rec, ebf, env0, nsteps):
    d = cls(p)
    d.env_enable(ep)
    d.set_envelope(env0)
    d.set_fields(ebf)
    d.set_species(0, rec)
    for it in range(1, nsteps + 1):
        d.env_run(it * p.dt, it)
    return d


@pytest.mark.parametrize("ndim,nx,ny,nz,n,how", CASES)
@pytest.mark.parametrize("pmax", [0.0, 2.0])
def test_env_tile_steps(ndim, nx, ny, nz, n, how, pmax):
    """Three envelope steps (the binning of one step serves the next): the
    density and current sums reach every output, so 1e-12 of the largest
    value (see above).  The tiles keep the records in another order: whole
    rows are compared, matched through each record's own weight."""
    from tests.test_envelope import env_case, numpy_init, pulse
    p, g, ep = env_case(ndim, nx=nx, ny=ny, nz=nz, der_ord=2, cap=n + 16, w_sh=10)
    env0 = numpy_init(p, pulse(p, a0=1.0, xc_frac=0.5, wx_frac=0.3, wy_frac=0.4))
    rec, ebf = records(p, n, how, pmax), 0.02 * laser_fields(p)
    wgh = 0.01 / max(n / 1000, 1) * (1 + np.arange(n) / n)  # one weight a record, FP32 numbers apart
    rec[:, 2 * ndim] = pack_slot(np.full(n, -1), np.zeros(n), wgh)
    assert np.unique(rec[:, 2 * ndim].view(np.uint64)).size == n
    dev = env_step(PicDevice, p, ep, rec, ebf, env0, 3)
    ora = env_step(Oracle, p, ep, rec, ebf, env0, 3)
    for f in ("get_envelope", "get_env_source", "get_fields", "get_currents"):
        a, b = getattr(dev, f)(), getattr(ora, f)()
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), f
    a, b = dev.get_species(0), ora.get_species(0)
    assert a.shape == b.shape
    a, b = (q[np.argsort(q[:, 2 * ndim].view(np.uint64))] for q in (np.ascontiguousarray(a), np.ascontiguousarray(b)))
    assert np.array_equal(a[:, 2 * ndim].view(np.uint64), b[:, 2 * ndim].view(np.uint64))
    for c in range(2 * ndim):
        assert np.abs(a[:, c] - b[:, c]).max() <= 1e-12 * np.abs(b[:, c]).max(), c


@pytest.mark.parametrize("ndim,nx,ny,nz", [(2, 33, 5, 1), (3, 33, 4, 4)])
def test_env_records_beyond_the_array(ndim, nx, ny, nz):
    """The last tiles reach beyond the field array.  A record placed out
    there is refused (index error), deposits nothing and is dropped, as in the
    per-particle kernels of the deterministic mode; a record outside the box
    whose stencil lies in the array counts.  Grids to 1e-12 (see above)."""
    from tests.test_envelope import env_case, numpy_init, pulse
    p, g, ep = env_case(ndim, nx=nx, ny=ny, nz=nz, cap=1000, w_sh=0)
    env0 = numpy_init(p, pulse(p, a0=1.0, xc_frac=0.5, wx_frac=0.3, wy_frac=0.4))
    rec = records(p, 300, "spread", 0.5)
    n, d, lo = [nx, ny, nz][:ndim], [p.dx, p.dy, p.dz], [p.gxmin, p.gymin, p.gzmin]
    top = [63.4, 7.4, 5.4]  # the tiles' last nodes
    k = 0
    for a in range(ndim):
        for far in (n[a] + 0.7, n[a] + 1.7, top[a]):  # above the box: within the array, beyond it, at the tiles' end
            rec[k, a] = lo[a] + far * d[a]
            k += 1
    for a in range(ndim):
        rec[k, a] = lo[a] + top[a] * d[a]
    rec[:, 2 * ndim] = pack_slot(np.full(300, -1), np.zeros(300), np.full(300, 0.05, np.float32))
    got = []
    for det in (False, True):
        dev = PicDevice(p)
        dev.env_enable(ep)
        dev.set_deterministic(det)
        dev.set_envelope(env0)
        dev.set_fields(0.02 * laser_fields(p))
        dev.set_species(0, rec)
        out = dev.env_run(p.dt, 1)
        assert out.error_bits & AGPU_EBIT_INDEX
        got.append((dev.get_envelope(), dev.get_env_source(), dev.get_fields(), dev.get_currents(),
                    sort_records(dev.get_species(0))))
        assert out.np[0] == got[-1][4].shape[0]
        dev.close()
    for a, b in zip(*got):
        assert a.shape == b.shape and np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
