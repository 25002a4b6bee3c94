"""Host transfers of the split form pass through a staging buffer in chunks
(agpu_set_species, agpu_get_species, agpu_window_inject, the field calls):
records and fields that take several chunks, and the device memory that the
calls leave in use."""
import numpy as np
import pytest

from aladyn_b200.abi import AGPU_FP32_SPLIT, AGPU_FP64
from aladyn_b200.sim import PicDevice
from tests.helpers import small_case
from tests.test_gpu_tiles import records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,nx,ny,nz,n", [(2, 5, 4, 1, 3001), (2, 301, 97, 1, 70001), (3, 33, 6, 7, 20011)])
def test_chunked_transfers(ndim, nx, ny, nz, n):
    """As many records as the capacity (five or seven chunks), the last third
    injected.  Split form: positions to 2^-25 cells (the offset's rounding) and
    the FP64 sums' own, momenta and weights as FP32, fields that are FP32
    numbers exactly."""
    p = small_case(ndim, nx=nx, ny=ny, nz=nz, cap=n, precision=AGPU_FP32_SPLIT)
    rec = records(p, n, "spread", 1.0)
    ebf = np.asfortranarray(np.random.default_rng(1).standard_normal(
        (nx + 5, ny + 5, nz + 5 if ndim == 3 else 1, p.nfield)).astype(np.float32).astype(np.float64))
    d = PicDevice(p)
    d.set_fields(ebf)
    d.set_species(0, rec[:n - n // 3])
    d.window_inject(0, rec[n - n // 3:])
    got = d.get_species(0)
    assert got.shape == rec.shape
    for a, cell in zip(range(ndim), (p.dx, p.dy, p.dz)):
        assert np.abs(got[:, a] - rec[:, a]).max() <= 2.0 ** -24 * cell
    assert np.array_equal(got[:, ndim:2 * ndim], rec[:, ndim:2 * ndim].astype(np.float32))
    assert np.array_equal(got[:, 2 * ndim].view(np.uint64), rec[:, 2 * ndim].view(np.uint64))
    assert np.array_equal(d.get_fields(), ebf)
    d.close()


@pytest.mark.parametrize("precision", [AGPU_FP32_SPLIT, AGPU_FP64])
def test_transfers_keep_no_memory(precision):
    """Transfers allocate nothing on the device that outlives them (the
    first handle loads the kernels)."""
    torch = pytest.importorskip("torch")
    p = small_case(2, nx=1000, ny=250, cap=1_000_000, precision=precision)
    rec = records(p, 1_000_000, "spread", 1.0)
    for rep in range(2):
        d = PicDevice(p)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        d.set_fields(np.zeros(d.field_shape(), order="F"))
        d.set_species(0, rec[:999_000])
        d.window_inject(0, rec[999_000:])
        d.get_species(0), d.get_fields(), d.get_currents()
        after = torch.cuda.mem_get_info()[0]
        d.close()
    assert after == before
