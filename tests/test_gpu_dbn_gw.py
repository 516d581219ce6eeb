"""GW-only differential number against the oracle at the edges of its tiles: redshift rows beyond one
staged group of 256, targets beyond one staged group of 512, unsorted targets (the reference stops at
the first one above the ISCO frequency), and targets that all lie above it."""

import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu

# a chain of about ten FP64 roundings and four powers of a 2-ulp pow(): below 40 ulp
RTOL = 40 * 2.2e-16


@pytest.mark.parametrize("nm,nq,nz,nf,order", [(2, 3, 1, 1, "up"), (5, 2, 257, 3, "up"), (3, 2, 7, 513, "up"),
                                               (6, 2, 31, 256, "mixed"), (4, 1, 9, 255, "high")])
def test_dbn_gw_tile_edges(built_lib, nm, nq, nz, nf, order):
    import torch
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam_cyutils
    rng = np.random.default_rng(nm * 1000 + nz + nf)
    mtot = np.logspace(np.log10(1e4 * C.MSOL), np.log10(1e12 * C.MSOL), nm)
    mrat = np.logspace(-3, 0, nq)
    zp = rng.uniform(0.001, 6.0, size=(nm, nq, nz))
    zp[rng.random(zp.shape) < 0.2] = -1.0
    dens = rng.lognormal(0.0, 3.0, size=zp.shape)
    dens[rng.random(zp.shape) < 0.1] = 0.0
    fobs = np.sort(10.0 ** rng.uniform(-9.0, -6.0, size=nf))
    if order == "mixed":     # the heavy cells' ISCO lies among these
        fobs = rng.permutation(10.0 ** rng.uniform(-9.0, -4.0, size=nf))
    elif order == "high":
        fobs = np.sort(10.0 ** rng.uniform(2.0, 3.0, size=nf))
    # one redshift per call: the reference's table walk carries its index from row to row, which is the
    # bracket only for rows in ascending order; these rows are in any order
    rows = [O.dbn_gw(fobs, dens[:, :, k:k + 1], mtot, mrat, zp[:, :, k:k + 1]) for k in range(nz)]
    rf, dn = (np.concatenate(x, axis=2) for x in zip(*rows))
    dev = [torch.as_tensor(x, device="cuda") for x in (fobs, dens, mtot, mrat, zp)]
    grf, gdn = (x.cpu().numpy() for x in sam_cyutils.dbn_gw_device(*dev))
    assert np.array_equal(grf, rf)
    assert np.array_equal(gdn == 0.0, dn == 0.0)
    np.testing.assert_allclose(gdn, dn, rtol=RTOL, atol=0)
