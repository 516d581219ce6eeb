"""The separation-step walk for ascending targets against the oracle at the edges of its tiles and rules:
redshift counts around one pass of 256 rows, targets around one, mrat counts off the cells of a block,
one step and many, duplicate targets, targets below and above every node, merger times beyond the age
of the Universe and at its end, and the FP64 walk (the same targets in descending order) beside it."""

import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu

# times agree to a few ulp and redshifts near z = 0 carry them as a difference (1e-16 of the age over
# dz = 1e-4); the residence time's powers magnify no further
RTOL = 1e-10


class _Hard:
    def __init__(self, norm, rchar, gi, go, steps, init):
        self._norm, self._rchar, self._gamma_inner, self._gamma_outer = norm, rchar, gi, go
        self._num_steps, self._sepa_init = steps, init

    def _norm_device(self):
        return self._norm


@pytest.mark.parametrize("nm,nq,nz,nf,steps,gi,seed", [
    (3, 2, 1, 1, 300, -1.0, 0), (2, 9, 7, 3, 300, -1.0, 1), (3, 3, 255, 4, 60, -0.7, 2), (2, 2, 257, 5, 300, -1.0, 3),
    (4, 17, 20, 40, 300, -1.0, 4), (2, 3, 11, 300, 100, 0.0, 5), (5, 4, 9, 20, 1, -1.0, 6), (2, 2, 5, 31, 2000, -1.0, 7)])
def test_walk_at_the_edges(built_lib, nm, nq, nz, nf, steps, gi, seed):
    import torch
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam_cyutils
    rng = np.random.default_rng(seed)
    mtot = np.logspace(np.log10(1e5 * C.MSOL), np.log10(1e11 * C.MSOL), nm)
    mrat = np.logspace(-2.5, 0, nq)
    redz = np.logspace(-3, 1, nz) if nz > 1 else np.array([0.4])
    gmt = 10.0 ** rng.uniform(-3.0, 1.2, size=(nm, nq, nz)) * C.GYR
    gmt.ravel()[::7] = 0.0
    dens = rng.lognormal(0.0, 2.0, size=gmt.shape)
    norm = 10.0 ** rng.uniform(6.5, 8.0, size=(nm, nq))
    fobs = np.sort(10.0 ** rng.uniform(-10.5, -7.0, size=nf))
    if nf > 4:
        fobs[nf // 2] = fobs[nf // 2 - 1]
        fobs[0], fobs[-1] = 1e-30, 1e3
    args = (1e3 * C.PC, steps, norm, 100.0 * C.PC, gi, 2.5, dens, mtot, mrat, redz, gmt)
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), device="cuda")
           for k, v in dict(norm=norm, dens=dens, mtot=mtot, mrat=mrat, redz=redz, gmt=gmt, up=fobs,
                            down=fobs[::-1].copy()).items()}
    hard = _Hard(dev["norm"], 100.0 * C.PC, gi, 2.5, steps, 1e3 * C.PC)
    for key in ("up", "down"):   # (the reference leaves a step at the first target past the last age)
        rf, dn = O.dbn_2pwl(dev[key].cpu().numpy(), *args)
        grf, gdn = (x.cpu().numpy() for x in sam_cyutils.dbn_2pwl_device(
            dev[key], hard, dev["dens"], dev["mtot"], dev["mrat"], dev["redz"], dev["gmt"]))
        assert np.array_equal(grf == -1.0, rf == -1.0), key
        assert np.array_equal(gdn == 0.0, dn == 0.0), key
        np.testing.assert_allclose(grf, rf, rtol=RTOL, atol=1e-13)
        np.testing.assert_allclose(gdn, dn, rtol=1e-8, atol=0)
