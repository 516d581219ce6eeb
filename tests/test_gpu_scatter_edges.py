"""The scatter's interpolation and redistribution at the edges of their tiles: regular grids that are not
a multiple of 32 nodes, slice counts off the kernels' groups of four and 26, scatter widths from one
that lets most of a row be passed over to one that needs it all, zero and huge densities, and rows
beyond the run mask.

The reference is a numpy restatement on the plan's own triangulation (points in order, one slice axis):
on some grids qhull keeps hull slivers that the plan peels off, so scipy's interpolant is another
function there."""

import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu


def _density(shape, seed):
    mtot, mrat, redz = O.grid_edges(shape)
    dens = O.static_binary_density(mtot, mrat, redz, O.default_params(scatter_dex=0.0))
    return mtot, mrat, dens * np.random.default_rng(seed).uniform(0.95, 1.05, size=dens.shape)


def _restated(mtot, mrat, dens, scatter, refine=4):
    from holodeck_gb300.sams import scatter as S
    a, sz = S.host_plan(mtot, mrat, scatter, refine)
    n, nz, N = sz.n_pts, dens.shape[2], sz.n_grid
    f = dens.reshape(n, nz)
    # minimum-norm-network gradients, Gauss-Seidel in point order, each slice to its own sweep
    g = np.zeros((n, 2, nz))
    open_ = np.ones(nz, bool)
    for _ in range(400):
        worst = np.zeros(nz)
        for i in range(n):
            sl = slice(a["nbr_ptr"][i], a["nbr_ptr"][i + 1])
            j, w = a["nbr_idx"][sl], a["nbr_w"][sl]
            c = 6.0 * (f[j] - f[i]) - 2.0 * np.einsum("ecz,ec->ez", g[j], w[:, :2])
            new = a["vtx_qinv"][i].reshape(2, 2) @ np.einsum("ez,ec->cz", c, w[:, 2:])
            change = np.abs(new - g[i]).max(axis=0) / np.maximum(1.0, np.abs(new).max(axis=0))
            worst = np.maximum(worst, np.where(open_, change, 0.0))
            g[i][:, open_] = new[:, open_]
        open_ &= worst >= 1e-6
        if not open_.any():
            break
    # Clough-Tocher with the plan's cross-derivative coefficients
    tri, lam, p = a["grid_tri"], a["grid_bary"], a["pts"]
    grid = np.full((N * N, nz), np.nan)
    for node in np.flatnonzero(tri >= 0):
        v = a["tri"][tri[node]]
        kap, P, F, G, L = a["tri_kappa"][tri[node]], p[v], f[v], g[v], lam[node]
        cen = P.mean(axis=0)
        ee = {(i, j): F[i] + (P[j] - P[i]) @ G[i] / 3.0 for i in range(3) for j in range(3) if i != j}
        al = [F[i] + (cen - P[i]) @ G[i] / 3.0 for i in range(3)]
        beta = []
        for k in range(3):
            i, j = (k + 1) % 3, (k + 2) % 3
            q20 = 3.0 * (al[i] - 0.5 * F[i] - 0.5 * ee[i, j])
            q02 = 3.0 * (al[j] - 0.5 * ee[j, i] - 0.5 * F[j])
            t20, t11, t02 = 3.0 * (ee[i, j] - F[i]), 3.0 * (ee[j, i] - ee[i, j]), 3.0 * (F[j] - ee[j, i])
            beta.append(0.5 * (ee[i, j] + ee[j, i]) +
                        (0.5 * (q20 + q02) + kap[k] * (t11 - 0.5 * (t20 + t02))) / 3.0)
        gam = [(al[i] + beta[(i + 1) % 3] + beta[(i + 2) % 3]) / 3.0 for i in range(3)]
        ctr = sum(gam) / 3.0
        k = int(np.argmin(L))
        i, j = (k + 1) % 3, (k + 2) % 3
        A, B, C = L[i] - L[k], L[j] - L[k], 3.0 * L[k]
        grid[node] = (F[i] * A ** 3 + F[j] * B ** 3 + ctr * C ** 3 + 3 * (ee[i, j] * A * A * B + ee[j, i] * A * B * B) +
                      3 * (al[i] * A * A * C + al[j] * B * B * C) + 3 * (gam[i] * A * C * C + gam[j] * B * C * C) +
                      6 * beta[k] * A * B * C)
    bad = ~(grid >= 0.0)
    grid = np.where(bad, f[a["grid_near"]], grid).reshape(N, N, nz)
    W = a["weights"]
    grid = np.einsum("jk,jbz->kbz", W @ W, grid)
    (ia, ib), (tx, ty) = a["back_idx"].T, a["back_t"].T[:, :, None]
    out = ((1 - tx) * ((1 - ty) * grid[ia, ib] + ty * grid[ia, ib + 1]) +
           tx * ((1 - ty) * grid[ia + 1, ib] + ty * grid[ia + 1, ib + 1]))
    return out.reshape(dens.shape)


@pytest.mark.parametrize("shape,scatter", [((9, 8, 1), 0.3), ((17, 11, 5), 0.05), ((24, 9, 27), 0.28),
                                           ((33, 12, 4), 0.9), ((10, 40, 3), 0.6)])
def test_scattered_density_against_restatement(built_lib, shape, scatter):
    from holodeck_gb300.sams import scatter as S
    mtot, mrat, dens = _density(shape, shape[0])
    ref = _restated(mtot, mrat, dens, scatter)
    got = S.add_scatter_to_masses(mtot, mrat, dens, scatter)
    big = ref > 1e-12 * ref.max()   # the tails carry the gradient solve's stopping tolerance
    np.testing.assert_allclose(got[big], ref[big], rtol=1e-9, atol=0)
    assert np.all(np.isfinite(got)) and np.all(got >= 0.0)


def test_zero_and_huge_slices(built_lib):
    """A slice is scattered by itself: zeros stay zero, and one slice's scale moves no other slice."""
    from holodeck_gb300.sams import scatter as S
    mtot, mrat, dens = _density((13, 10, 6), 1)
    want = S.add_scatter_to_masses(mtot, mrat, dens, 0.3)
    odd = dens.copy()
    odd[:, :, 2] = 0.0
    odd[:, :, 4] *= 2.0 ** 400
    got = S.add_scatter_to_masses(mtot, mrat, odd, 0.3)
    assert np.all(got[:, :, 2] == 0.0)
    assert np.array_equal(got[:, :, [0, 1, 3, 5]], want[:, :, [0, 1, 3, 5]])
    assert np.all(np.isfinite(got[:, :, 4])) and np.all(got[:, :, 4] > 0.0)


def test_rows_beyond_the_run_mask(built_lib):
    """refine = 16 gives 1056 nodes a row (33 runs), summed in full."""
    from holodeck_gb300.sams import scatter as S
    mtot, mrat, dens = _density((66, 5, 2), 3)
    got = S.add_scatter_to_masses(mtot, mrat, dens, 0.3, refine=16)
    ref = _restated(mtot, mrat, dens, 0.3, refine=16)
    big = ref > 1e-10 * ref.max()
    np.testing.assert_allclose(got[big], ref[big], rtol=1e-8, atol=0)
