"""Arrays of a caller off a 16-byte boundary: the scatter's workspace and plan, the strain's distance cubics."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(x, by):
    """The same values in device memory `by` bytes off a 16-byte boundary (and the storage that holds them)."""
    import torch
    pad = by // x.element_size()
    hold = torch.empty(x.numel() + 8, dtype=x.dtype, device=x.device)
    view = hold[pad:pad + x.numel()]
    view.copy_(x.reshape(-1))
    assert view.data_ptr() % 16 == by
    return view


@pytest.mark.parametrize("what", ["workspace", "ph_ptr", "ph_info", "ph_m"])
def test_scatter(built_lib, what):
    import torch
    from holodeck_gb300 import _device as D, _native as N
    from holodeck_gb300.sams import scatter as S
    rng = np.random.default_rng(2)
    mtot, mrat, nz = np.logspace(38, 44, 12), np.logspace(-3, 0, 9), 5
    dens = torch.as_tensor(rng.lognormal(0.0, 1.0, size=(12, 9, nz)), device="cuda")
    want = S.add_scatter_to_masses_device(mtot, mrat, dens.clone(), 0.3)
    plan = S.DevicePlan(mtot, mrat, 0.3)
    if what != "workspace":
        by = 8 if what == "ph_m" else 4
        hold = _shifted(plan.dev[what], by)
        setattr(plan.struct, what, N.ptr(hold))
    bytes_ = int(N.load().hgb_scatter_workspace_bytes(12, 9, nz, plan.struct.n_grid))
    ws = torch.empty(bytes_ // 8 + 2, dtype=torch.float64, device="cuda")
    assert ws.data_ptr() % 16 == 0
    at = ws.data_ptr() + (8 if what == "workspace" else 0)
    got, st = dens.clone(), D.StatusWord()
    N.call("hgb_add_scatter_to_masses", ctypes.byref(plan.struct), N.ptr(got), nz, at, bytes_, st.ptr, N.stream_handle())
    assert st.read() == 0
    # another plan's order of sums (sweeps one after another) leaves rounding inside the solve's tolerance
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=0.0 if what == "workspace" else 1e-9)


def test_strain_without_aligned_cubics(built_lib):
    import torch
    from holodeck_gb300 import _device as D, _native as N, constants as C
    from holodeck_gb300.cosmology import cosmo
    mt, mr, fe = D.as_devices(np.logspace(38, 44, 4), np.logspace(-2, 0, 3), np.linspace(1.0, 6.0, 6) * 1e-9)
    rz = torch.as_tensor(np.random.default_rng(1).uniform(0.01, 6.0, size=(4, 3, 7, 5)), device="cuda")

    def strain(dc):
        out, st = torch.empty((3, 2, 6, 5), dtype=torch.float64, device="cuda"), D.StatusWord()
        N.call("hgb_char_strain_sq", N.ptr(mt), 4, N.ptr(mr), 3, 7, N.ptr(fe), 5, N.ptr(rz), C.GW_SRC_CONST, dc.ref,
               N.ptr(out), st.ptr, N.stream_handle())
        assert st.read() == 0
        return out

    null, off = D.DeviceCosmology(cosmo), D.DeviceCosmology(cosmo)
    null.struct.dc_cub = None
    hold = _shifted(off.dc_cub, 8)
    off.struct.dc_cub = N.ptr(hold)
    assert torch.equal(strain(off), strain(null))
