"""The walk for ascending targets on rows without ascending times: a normalisation, mass, redshift, merger time
or target that is NaN, negative, zero or infinite, and a start inside the ISCO.  The walk for targets in any
order, given the same ascending targets, is the measure: where it has a NaN or no bracket, so has this one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NM, NQ, NZ, NF, STEPS = 3, 9, 11, 7, 120


def _inputs(case):
    from holodeck_gb300 import constants as C
    rng = np.random.default_rng(5)
    a = dict(mtot=np.logspace(7, 10, NM) * C.MSOL, mrat=np.logspace(-2, 0, NQ), redz=np.linspace(0.05, 3.0, NZ),
             gmt=10.0 ** rng.uniform(-3.0, 0.3, size=(NM, NQ, NZ)) * C.GYR, norm=10.0 ** rng.uniform(6.5, 7.5, size=(NM, NQ)),
             fobs=np.logspace(-9.5, -8.0, NF), init=1e3 * C.PC)
    if case == "norm":
        a["norm"][0, 0], a["norm"][1, 4], a["norm"][2, 7], a["norm"][0, 8] = np.nan, -1e7, np.inf, 0.0
    elif case == "no_rate":   # no hardening and no GW emission: steps without an end
        a["norm"][1, 0], a["mrat"][0] = 0.0, 0.0
    elif case == "mass":
        a["mtot"][1] = np.nan
    elif case == "ratio":
        a["mrat"][2], a["mrat"][5] = np.nan, -0.5
    elif case == "redz":
        a["redz"][3] = np.nan
    elif case == "gmt":
        a["gmt"][0, 1, 2], a["gmt"][1, 2, 3], a["gmt"][2, 3, 4], a["gmt"][2, 8, 10] = np.nan, -0.3 * C.GYR, np.inf, -np.inf
    elif case == "target":
        a["fobs"] = np.array([np.nan])
    elif case == "inside":
        a["init"], a["fobs"] = 1e-5 * C.PC, np.logspace(-5.5, -3.5, NF)   # the ISCO of two masses lies further out
    return a


@pytest.mark.parametrize("case", ["plain", "norm", "no_rate", "mass", "ratio", "redz", "gmt", "target", "inside"])
def test_rows_without_ascending_times(built_lib, case):
    import torch
    from holodeck_gb300 import _device as D, _native as N, constants as C
    from holodeck_gb300.cosmology import cosmo
    a = _inputs(case)
    dev = {k: torch.as_tensor(v, device="cuda") for k, v in a.items() if k != "init"}
    dens = torch.ones((NM, NQ, NZ), dtype=torch.float64, device="cuda")
    dc = D.device_cosmology(cosmo)
    nf = a["fobs"].size
    got = []
    for ascending in (1, 0):
        out = [torch.full((NM, NQ, NZ, nf), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
        N.call("hgb_dbn_2pwl_phase", N.ptr(dev["fobs"]), nf, ascending, a["init"], STEPS, N.ptr(dev["norm"]), 100.0 * C.PC,
               -1.0, 2.5, N.ptr(dens), N.ptr(dev["mtot"]), NM, N.ptr(dev["mrat"]), NQ, N.ptr(dev["redz"]), NZ,
               N.ptr(dev["gmt"]), dc.ref, N.ptr(out[0]), N.ptr(out[1]), 3, N.stream_handle())
        got.append([x.cpu().numpy() for x in out])
    (rf, dn), (want_rf, want_dn) = got
    assert np.array_equal(np.isnan(dn), np.isnan(want_dn))
    assert np.array_equal(rf == -1.0, want_rf == -1.0)
    assert np.array_equal(dn == 0.0, want_dn == 0.0)
    # as in test_gpu_walk_edges: times to a few ulp, and what a difference near z = 0 makes of them
    np.testing.assert_allclose(rf, want_rf, rtol=1e-10, atol=1e-13)
    np.testing.assert_allclose(dn, want_dn, rtol=1e-8, atol=0)


@pytest.mark.parametrize("dens", [1e-290, 1e-303, 1e-308, 1e-312])
def test_least_densities(built_lib, dens):
    """A number is its density times a factor that does not depend on it, down to the subnormals."""
    import types
    import torch
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam_cyutils
    a = _inputs("plain")
    dev = {k: torch.as_tensor(v, device="cuda") for k, v in a.items() if k != "init"}
    hard = types.SimpleNamespace(_sepa_init=a["init"], _num_steps=STEPS, _rchar=100.0 * C.PC, _gamma_inner=-1.0,
                                 _gamma_outer=2.5, _norm_device=lambda: dev["norm"])

    def number(value):
        nden = torch.full((NM, NQ, NZ), value, dtype=torch.float64, device="cuda")
        return sam_cyutils.dbn_2pwl_device(dev["fobs"], hard, nden, dev["mtot"], dev["mrat"], dev["redz"],
                                           dev["gmt"])[1].cpu().numpy()

    one, got = number(1.0), number(dens)
    assert (one > 0.0).sum() > 100
    # the density times a factor of one and a half ulp, in two roundings, and a step of the subnormals
    assert np.all(np.abs(got - dens * one) <= 8e-16 * (dens * one) + 1e-323)
