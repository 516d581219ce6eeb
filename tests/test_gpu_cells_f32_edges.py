"""FP32 cell integration and strain against the FP64 kernel at the edges of its redshift runs: frequency
counts around a warp and up to one thread each, short and empty runs, sentinels mixed with redshifts.

Number: eight truncated vertices (2^-23), the compensated sum, two truncated factors and three products,
below 1e-6.  Strain: at worst 2.5e-6 in its root (powf 4, the divisions 2 + 2 + 2, rcbrtf 1 units of 2^-23,
the table's Hermite sum and the products the rest), 6e-6 squared, and the FP64 kernel's own 8e-14 / z."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(nm, nq, nz, nf, seed):
    from holodeck_gb300 import constants as C
    rng = np.random.default_rng(seed)
    mtot = np.logspace(np.log10(1e5 * C.MSOL), np.log10(1e11 * C.MSOL), nm)
    mrat, redz = np.logspace(-2.5, 0, nq), np.logspace(-3, 1, nz)
    fe = np.linspace(0.5, nf + 0.5, nf + 1) / (32.0 * C.YR)
    shape = (nm, nq, nz, nf)
    rf = rng.uniform(0.002, 8.0, size=shape)
    rf[rng.random(shape) < 0.1] = -1.0
    rf[rng.random(shape) < 0.05] = 0.0
    rf[..., : nf // 3] = -1.0
    dn = rng.lognormal(0.0, 5.0, size=shape) * (rf >= 0.0)
    return mtot, mrat, redz, fe, rf, dn


@pytest.mark.parametrize("nm,nq,nz,nf", [(2, 2, 2, 1), (3, 2, 3, 31), (2, 3, 40, 33), (2, 2, 9, 255), (2, 2, 4, 256),
                                         (2, 2, 5, 129), (3, 3, 300, 2), (4, 3, 7, 40)])
def test_f32_cells_at_the_edges(built_lib, nm, nq, nz, nf):
    import torch
    from holodeck_gb300 import _device as D
    from holodeck_gb300 import _native as N
    from holodeck_gb300 import constants as C
    from holodeck_gb300.cosmology import cosmo
    mtot, mrat, redz, fe, rf, dn = _inputs(nm, nq, nz, nf, nm * 1000 + nz)
    dc = D.device_cosmology(cosmo, torch.device("cuda", 0))
    dev = [D.as_device(x) for x in (mtot, np.log10(mtot), mrat, redz, fe, np.diff(np.log(fe)), dn, rf)]

    def cells(fn):
        number = torch.full((nm - 1, nq - 1, nz - 1, nf), -7.0, dtype=torch.float64, device="cuda")
        h2 = number.clone()
        st = D.StatusWord()
        N.call(fn, N.ptr(dev[0]), N.ptr(dev[1]), nm, N.ptr(dev[2]), nq, N.ptr(dev[3]), nz, N.ptr(dev[4]),
               N.ptr(dev[5]), nf, N.ptr(dev[6]), N.ptr(dev[7]), C.GW_SRC_CONST, dc.ref, N.ptr(number), N.ptr(h2),
               st.ptr, N.stream_handle())
        assert st.read() == 0
        return number.cpu().numpy(), h2.cpu().numpy()

    n64, h64 = cells("hgb_number_and_strain")
    n32, h32 = cells("hgb_number_and_strain_f32")
    assert np.array_equal(n32 == 0.0, n64 == 0.0) and np.array_equal(h32 == 0.0, h64 == 0.0)
    assert np.all(np.abs(n32 - n64) <= 1e-6 * n64)
    mid = rf
    for axis in range(3):
        n = mid.shape[axis]
        mid = 0.5 * (np.take(mid, range(1, n), axis) + np.take(mid, range(n - 1), axis))
    z = np.clip(mid, 1e-300, None)
    assert np.all(np.abs(h32 - h64) <= (6e-6 + 8e-14 / z) * h64)
