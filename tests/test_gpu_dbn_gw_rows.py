"""GW-only differential number where a block's rows lie in many cells, in parts of cells and in one cell, against
the oracle; and grids of few redshifts next to grids of many with the same number of points."""
import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu

# a chain of about ten FP64 roundings and four powers of a 2-ulp pow(): below 40 ulp
RTOL = 40 * 2.2e-16


def _inputs(nm, nq, nz, nf):
    from holodeck_gb300 import constants as C
    rng = np.random.default_rng(nm * 1000 + nz + nf)
    mtot = np.logspace(np.log10(1e4 * C.MSOL), np.log10(1e12 * C.MSOL), nm)
    mrat = np.logspace(-3, 0, nq)
    zp = rng.uniform(0.001, 6.0, size=(nm, nq, nz))
    zp[rng.random(zp.shape) < 0.2] = -1.0
    return np.sort(10.0 ** rng.uniform(-9.0, -5.0, size=nf)), rng.lognormal(0.0, 3.0, size=zp.shape), mtot, mrat, zp


@pytest.mark.parametrize("nm,nq,nz,nf", [(1, 1, 1, 1), (2, 1, 300, 3), (40, 31, 1, 2), (181, 161, 1, 1), (181, 161, 2, 3),
                                         (91, 81, 3, 2), (61, 47, 53, 5), (70, 67, 33, 1), (9, 8, 8, 515)])
def test_rows_across_cells(built_lib, nm, nq, nz, nf):
    import torch
    from holodeck_gb300.sams import sam_cyutils
    fobs, dens, mtot, mrat, zp = _inputs(nm, nq, nz, nf)
    # one redshift per call: the reference's table walk is the bracket only for rows in ascending order
    rows = [O.dbn_gw(fobs, dens[:, :, k:k + 1], mtot, mrat, zp[:, :, k:k + 1]) for k in range(nz)]
    rf, dn = (np.concatenate(x, axis=2) for x in zip(*rows))
    dev = [torch.as_tensor(x, device="cuda") for x in (fobs, dens, mtot, mrat, zp)]
    grf, gdn = (x.cpu().numpy() for x in sam_cyutils.dbn_gw_device(*dev))
    assert np.array_equal(grf, rf)
    assert np.array_equal(gdn == 0.0, dn == 0.0)
    np.testing.assert_allclose(gdn, dn, rtol=RTOL, atol=0)


def test_few_redshifts_cost_what_many_do(built_lib):
    """The same points as many cells of one redshift: within four times the time of few cells of many (a block
    per cell took more than ten)."""
    import torch
    from holodeck_gb300.sams import sam_cyutils
    best = []
    for shape in ((300, 300, 1), (30, 30, 100)):
        dev = [torch.as_tensor(x, device="cuda") for x in _inputs(*shape, 1)]
        times = []
        for _ in range(12):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            begin.record()
            sam_cyutils.dbn_gw_device(*dev)
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        best.append(min(times))
    assert best[0] < 4.0 * best[1], best


@pytest.mark.parametrize("dens", [1e-300, 1e-305, 1e-310, 5e-324])
def test_least_densities(built_lib, dens):
    """Densities down to the least double keep their bits: RTOL of the value and a step of the subnormals."""
    import torch
    from holodeck_gb300.sams import sam_cyutils
    fobs, like, mtot, mrat, zp = _inputs(7, 5, 1, 9)
    full = np.full(like.shape, dens)
    rf, dn = O.dbn_gw(fobs, full, mtot, mrat, zp)
    dev = [torch.as_tensor(x, device="cuda") for x in (fobs, full, mtot, mrat, zp)]
    grf, gdn = (x.cpu().numpy() for x in sam_cyutils.dbn_gw_device(*dev))
    assert np.array_equal(grf, rf) and dn.max() > 0.0
    # the reference rounds to a subnormal once or twice on its way, each half a step of what follows
    slack = 5e-324 * (2.0 + dn / dens)
    assert np.all(np.abs(gdn - dn) <= RTOL * dn + slack)
