"""Cell integration and strain with the elements of a cell shared out in every way the rule makes: short and
full warps of frequencies, two passes over them, one and several blocks a cell.  A bin's value does not depend
on its neighbours, so each way gives the bits of the bins taken a few frequencies and redshifts at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(model, mtot, mrat, redz, fe, dn, rf, precision):
    from holodeck_gb300 import _device as D
    model.mtot, model.mrat, model.redz = mtot, mrat, redz
    model._edges_t = None
    st = D.StatusWord()
    out = model._number_and_strain(fe, dn.contiguous(), rf.contiguous(), status=st, precision=precision)
    assert st.read() == 0
    return out


@pytest.mark.parametrize("nm,nq,nz,nf", [(2, 2, 2, 1), (2, 2, 601, 1), (3, 2, 90, 33), (3, 3, 301, 129), (2, 3, 40, 255),
                                         (40, 31, 3, 3), (3, 3, 61, 257), (2, 2, 301, 300), (30, 30, 17, 86)])
def test_every_split_gives_the_same_bits(built_lib, nm, nq, nz, nf):
    import torch
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam as S, sam_cyutils
    rng = np.random.default_rng(nz + nf)
    mtot, mrat, redz = np.logspace(38, 44, nm), np.logspace(-2, 0, nq), np.logspace(-3, 1, nz)
    fe = np.linspace(0.5, nf + 0.5, nf + 1) / (32.0 * C.YR)
    rf = torch.as_tensor(rng.uniform(0.002, 8.0, size=(nm, nq, nz, nf)), device="cuda")
    dn = torch.as_tensor(rng.lognormal(0.0, 5.0, size=rf.shape), device="cuda")
    gone = torch.as_tensor(rng.random(rf.shape) < 0.1, device="cuda")
    rf[gone], dn[gone] = -1.0, 0.0
    model = S.Semi_Analytic_Model(shape=(nm, nq, nz))
    for precision in ("fp64",) + (("fp32",) if nf <= 256 else ()):
        number, h2 = _cells(model, mtot, mrat, redz, fe, dn, rf, precision)
        for f0, f1 in ((0, min(nf, 7)), (nf // 2, nf // 2 + 1), (max(0, nf - 5), nf)):
            for z0, z1 in ((0, min(nz, 4)), (max(0, nz - 3), nz), (nz // 3, min(nz, nz // 3 + 12))):
                if z1 - z0 < 2:
                    continue
                part = S.Semi_Analytic_Model(shape=(nm, nq, z1 - z0))
                n, h = _cells(part, mtot, mrat, redz[z0:z1], fe[f0:f1 + 1], dn[:, :, z0:z1, f0:f1],
                              rf[:, :, z0:z1, f0:f1], precision)
                assert torch.equal(number[:, :, z0:z1 - 1, f0:f1], n)
                assert torch.equal(h2[:, :, z0:z1 - 1, f0:f1], h)
        if precision == "fp64":
            assert torch.equal(sam_cyutils.integrate_device([mtot, mrat, redz, fe], dn), number)
