"""The phases in which the scatter's gradient solve runs several Gauss-Seidel sweeps at once: the plan's
arrays, and the pipelined schedule on the CPU against sweeps one after another; on the GPU, the
pipelined kernel against the one that takes a level at a time."""

import ctypes

import numpy as np
import pytest

from oracle import sam_oracle as O

SHAPES = [(2, 2), (2, 9), (9, 2), (10, 11), (14, 13), (24, 60), (60, 8)]


def _plan(shape):
    from holodeck_gb300.sams import scatter as S
    mtot, mrat, _ = O.grid_edges(shape + (3,))
    return (mtot, mrat) + S.host_plan(mtot, mrat, 0.3)


def _entries(arrs, p, few):
    """Positions of point p's entries in ph_nbr / ph_m."""
    _, _, deg, off = arrs["ph_info"][p]
    return off + np.arange(deg) * (few if deg <= 8 else 1)


@pytest.mark.parametrize("shape", SHAPES)
def test_pipelined_sweeps_read_what_sequential_sweeps_read(built_lib, shape):
    mtot, mrat, a, sz = _plan(shape)
    n = shape[0] * shape[1]
    nph, nlev = sz.n_phases, sz.n_levels
    assert 1 <= nph <= n and (nlev - 1) // nph < 8
    info, ptr, nbr = a["ph_info"], a["ph_ptr"], a["nbr_ptr"]
    assert sorted(info[:, 0]) == list(range(n))
    assert sz.phase_width == ptr[:, 1].max()
    few_of = np.empty(n, int)
    entries = []
    for f in range(nph):
        start, cnt, few, _ = ptr[f]
        assert start == (0 if f == 0 else ptr[f - 1, :2].sum()) and 0 <= few <= cnt
        deg = info[start:start + cnt, 2]
        assert np.all(deg[:few] <= 8) and np.all(deg[few:] > 8)
        few_of[start:start + cnt] = few
    pos = np.empty(n, int)
    pos[info[:, 0]] = np.arange(n)
    for p in range(n):
        k = _entries(a, p, few_of[p])
        assert k.size == 0 or (k.min() >= 0 and k.max() < a["ph_nbr"].size)
        entries.append(k)
        i = info[p, 0]
        assert np.array_equal(a["ph_nbr"][k], pos[a["nbr_idx"][nbr[i]:nbr[i + 1]]])
    used = np.concatenate(entries)
    assert np.unique(used).size == used.size
    # the schedule: random right-hand sides, sweeps one after another and in phases
    rng = np.random.default_rng(n)
    c = rng.normal(size=(n, 2))
    sweeps = 5
    order = np.arange(n)[np.argsort(info[:, 0])]      # positions in point order
    seq, g = [], np.zeros((n, 2))
    for _ in range(sweeps):
        for p in order:
            m = a["ph_m"][entries[p]].reshape(-1, 2, 2)
            g[p] = c[p] + np.einsum("eij,ej->i", m, g[a["ph_nbr"][entries[p]]])
        seq.append(g.copy())
    g, got = np.zeros((n, 2)), np.full((sweeps, n, 2), np.nan)
    for T in range(sweeps + (nlev - 1) // nph):
        for f in range(nph):
            members = np.arange(ptr[f, 0], ptr[f, 0] + ptr[f, 1])
            new = {}
            for p in members:
                k = T - info[p, 1]
                if 0 <= k < sweeps:
                    m = a["ph_m"][entries[p]].reshape(-1, 2, 2)
                    new[p] = c[p] + np.einsum("eij,ej->i", m, g[a["ph_nbr"][entries[p]]])
                    got[k, p] = new[p]
            for p, v in new.items():
                g[p] = v
    assert np.array_equal(got, np.array(seq))


@pytest.mark.parametrize("shape", [(9, 7), (31, 17)])
def test_update_matrices_are_the_normal_equations(built_lib, shape):
    """c_i + sum_j M_ij g_j equals Q^-1 sum_j (6 (f_j - f_i) - 2 g_j . w01) w23."""
    _, _, a, _ = _plan(shape)
    n = shape[0] * shape[1]
    rng = np.random.default_rng(n)
    f, g = rng.normal(size=n), rng.normal(size=(n, 2))
    few_of = np.repeat(a["ph_ptr"][:, 2], a["ph_ptr"][:, 1])
    gp = g[a["ph_info"][:, 0]]
    for p in range(n):
        i = a["ph_info"][p, 0]
        sl = slice(a["nbr_ptr"][i], a["nbr_ptr"][i + 1])
        j, w, q = a["nbr_idx"][sl], a["nbr_w"][sl], a["vtx_qinv"][i].reshape(2, 2)
        want = q @ (((6.0 * (f[j] - f[i]) - 2.0 * (g[j] * w[:, :2]).sum(axis=1))[:, None] * w[:, 2:]).sum(axis=0))
        k = _entries(a, p, few_of[p])
        got = q @ (6.0 * (f[j] - f[i])[:, None] * w[:, 2:]).sum(axis=0)
        got = got + np.einsum("eij,ej->i", a["ph_m"][k].reshape(-1, 2, 2), gp[a["ph_nbr"][k]])
        scale = np.abs(q) @ (np.abs(w[:, 2:]) * (6.0 * np.abs(f[j] - f[i]) + 2.0 * np.abs(g[j] * w[:, :2]).sum(axis=1))[
            :, None]).sum(axis=0)
        assert np.all(np.abs(got - want) <= 40 * 2.2e-16 * scale)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nz,maxiter", [((3, 2), 1, 400), ((10, 11), 33, 400), ((24, 60), 5, 400),
                                              ((60, 8), 3, 3), ((91, 81), 2, 400), ((140, 110), 2, 400),
                                              ((140, 110), 1, 1)])
def test_pipelined_solve_matches_level_by_level(built_lib, shape, nz, maxiter):
    """Densities scattered with the phases, and with a plan without them (one level at a time); the
    largest grids keep their gradients outside shared memory.  A gradient's regrouped sum moves it by a
    few ulp per sweep; the scattered density is a positive average of the interpolant."""
    import torch
    from holodeck_gb300 import _device as D
    from holodeck_gb300 import _native as N
    from holodeck_gb300.sams import scatter as S
    mtot, mrat, _ = O.grid_edges(shape + (3,))
    m1 = mtot[:, None, None] / (1.0 + mrat[None, :, None])
    rng = np.random.default_rng(shape[0])
    z = np.linspace(0.0, 1.0, nz)
    dens = 1e-3 * (m1 / m1.min()) ** -0.3 * np.exp(-m1 / m1.max() * 20.0) * (1.0 + mrat[None, :, None]) * (2.0 - z)
    dens = dens * rng.uniform(0.9, 1.1, size=dens.shape)
    plan = S.device_plan(mtot, mrat, 0.3)
    out, codes = [], []
    for phases in (True, False):
        struct = N.HgbScatterPlan.from_buffer_copy(plan.struct)
        struct.grad_maxiter = maxiter
        if not phases:
            struct.ph_ptr = None
        d = torch.as_tensor(dens, device="cuda").contiguous()
        ws_bytes = N.load().hgb_scatter_workspace_bytes(shape[0], shape[1], nz, plan.sizes.n_grid)
        ws = D.workspace(ws_bytes, d.device)
        st = D.StatusWord(d.device)
        N.call("hgb_add_scatter_to_masses", ctypes.byref(struct), N.ptr(d), nz, N.ptr(ws), int(ws_bytes), st.ptr,
               N.stream_handle())
        codes.append(st.read())
        out.append(d.cpu().numpy())
    assert codes[0] == codes[1]
    assert np.all(np.isfinite(out[0]))
    np.testing.assert_allclose(out[0], out[1], rtol=1e-11, atol=0)
