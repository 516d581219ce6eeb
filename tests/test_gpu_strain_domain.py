"""Strain outside the domain of its fractional powers: NaN, as the reference's powers give it, not the finite
value of a cube root."""
import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["mtot", "mrat", "fobs", "zero"])
def test_negative_edges(built_lib, which):
    from holodeck_gb300 import gravwaves
    mtot, mrat, redz = np.logspace(40, 43, 4), np.logspace(-2, 0, 4), np.linspace(0.1, 2.0, 5)
    fe = np.linspace(1.0, 6.0, 6) * 1e-9
    if which == "mtot":
        mtot[:2] *= -1.0
    elif which == "mrat":
        mrat[:2] = -0.3, -0.2
    elif which == "fobs":
        fe = np.linspace(-2.5, 2.5, 6) * 1e-9
    else:
        mtot[:2], mrat[:2] = 0.0, 0.0
    rf = np.random.default_rng(0).uniform(0.05, 2.0, size=(4, 4, 5, 5))
    rf[:, :, 0] = -1.0
    with np.errstate(all="ignore"):
        want = O.char_strain_sq_from_bin_edges_redz([mtot, mrat, redz, fe], rf)
    mid = rf
    for axis in range(3):
        mid = 0.5 * (np.take(mid, range(1, mid.shape[axis]), axis) + np.take(mid, range(mid.shape[axis] - 1), axis))
    want[mid <= 0.0] = 0.0   # no binaries there, whatever the edges
    got = gravwaves.char_strain_sq_from_bin_edges_redz([mtot, mrat, redz, fe], rf)
    assert np.isnan(want).any() == (which != "zero")
    assert np.array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_allclose(got, want, rtol=1e-11)   # 4e-14 / z of the distance at z > 0.01
