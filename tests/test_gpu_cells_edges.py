"""Cell integration and strain against the oracle at the edges of their tiles: frequency counts around a
warp and around one block, redshift counts that leave runs short or empty, single cells, midpoints that
mix the -1 sentinel with redshifts (down to z ~ 1e-7), zeros, and a distance table whose size is no
power of two (the general lookup)."""

import numpy as np
import pytest

from oracle import sam_oracle as O

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
    if nz > 2:   # corners whose mean with a sentinel nearly cancels
        rf[:, :, 0, -1] = -1.0
        rf[:, :, 1, -1] = 1.0 + 4e-6 * rng.random(shape[:2])
    dn = rng.lognormal(0.0, 5.0, size=shape) * (rf >= 0.0)
    return [mtot, mrat, redz, fe], rf, dn


@pytest.mark.parametrize("nm,nq,nz,nf", [(2, 2, 2, 1), (3, 2, 3, 31), (2, 3, 40, 33), (2, 2, 9, 255), (2, 2, 4, 257),
                                         (3, 3, 300, 2), (4, 3, 7, 40)])
def test_cells_at_the_edges(built_lib, nm, nq, nz, nf):
    from holodeck_gb300 import gravwaves
    from holodeck_gb300.sams import sam_cyutils
    edges, rf, dn = _inputs(nm, nq, nz, nf, nm * 1000 + nz)
    number = sam_cyutils.integrate_differential_number_3dx1d(edges, dn)
    assert np.array_equal(number, O.integrate_differential_number_3dx1d(edges, dn))
    h2 = gravwaves.char_strain_sq_from_bin_edges_redz(edges, rf)
    want = O.char_strain_sq_from_bin_edges_redz(edges, rf)
    assert np.array_equal(h2 == 0.0, want == 0.0)
    # u = (1 + z)^(-1/2) carries 1e-14 into the distance's 1 - u ~ z / 2: 4e-14 / z in the strain squared
    z = np.clip(_mid(_mid(_mid(rf, 0), 1), 2), 1e-300, None)
    assert np.all(np.abs(h2 - want) <= (1e-12 + 8e-14 / z) * want)


def _mid(x, axis):
    return 0.5 * (np.take(x, range(1, x.shape[axis]), axis) + np.take(x, range(x.shape[axis] - 1), axis))


def test_general_distance_table(built_lib):
    """A table without cubics, and one of 3000 intervals, take the general lookup: the same strain to the
    tables' own error."""
    import torch
    from holodeck_gb300 import _device as D
    from holodeck_gb300 import _native as N
    from holodeck_gb300 import constants as C
    from holodeck_gb300.cosmology import cosmo
    edges, rf, _ = _inputs(4, 3, 7, 5, 1)
    mt, mr, fe, r = (D.as_device(x) for x in (edges[0], edges[1], edges[3], rf))

    def strain(dc):
        out = torch.empty((3, 2, 6, 5), dtype=torch.float64, device="cuda")
        st = D.StatusWord()
        N.call("hgb_char_strain_sq", N.ptr(mt), 4, N.ptr(mr), 3, 7, N.ptr(fe), 5, N.ptr(r), C.GW_SRC_CONST, dc.ref,
               N.ptr(out), st.ptr, N.stream_handle())
        assert st.read() == 0
        return out.cpu().numpy()

    want = strain(D.DeviceCosmology(cosmo))
    plain = D.DeviceCosmology(cosmo)
    plain.struct.dc_cub = None
    np.testing.assert_allclose(strain(plain), want, rtol=1e-9)
    other = D.DeviceCosmology(cosmo)
    val, der = D.comoving_distance_table(cosmo, 3000)
    keep = [D.as_device(val), D.as_device(der), D.as_device(D.distance_cubics(val, der, 3000))]
    other.struct.dc_n = 3000
    other.struct.dc_val, other.struct.dc_der, other.struct.dc_cub = (N.ptr(x) for x in keep)
    big = want > 0.0
    big &= _mid(_mid(_mid(rf, 0), 1), 2) > 1e-3   # the coarser table's error grows towards z = 0
    np.testing.assert_allclose(strain(other)[big], want[big], rtol=1e-9)
