"""The parameter grids' scale exponents, gathered by blocks: numpy's frexp of the largest finite magnitude over
the bins with strain, at sizes around a block and with bins that have no redshift, no strain, or neither."""
import numpy as np
import pytest
import torch

from holodeck_gb300 import constants as C
from holodeck_gb300 import single_sources as SS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2, 1), (2, 2, 9, 32), (3, 2, 5, 31), (2, 2, 2, 257), (5, 4, 7, 40)])
@pytest.mark.parametrize("kind", ["mixed", "none", "near"])
def test_scales(shape, kind):
    nm, nq, nz, nf = shape
    rng = np.random.default_rng(nz * nf)
    edges = [np.logspace(6, 10, nm) * C.MSOL, np.logspace(-2, 0, nq), np.logspace(-2, 1, nz),
             np.linspace(0.5, nf + 0.5, nf + 1) / (32.0 * C.YR)]
    rz = rng.uniform(0.01, 6.0, shape)
    if kind == "near":
        rz = rz * 1e-310   # subnormal redshifts
    rz[rng.random(shape) < 0.2] = -1.0
    if kind == "none":
        rz[:] = -1.0
    bins = (nm - 1, nq - 1, nz - 1, nf)
    h2 = rng.uniform(1e-34, 1e-30, bins) * (rng.random(bins) < 0.7)
    grids, scales = SS.param_grids_device(edges, torch.as_tensor(rz, device="cuda"), h2fdf=torch.as_tensor(h2, device="cuda"))
    scales = scales.cpu().numpy()
    for k, g in enumerate(grids):
        v = np.abs(g.cpu().numpy()[h2 != 0.0])
        v = v[np.isfinite(v) & (v > 0.0)]
        want = np.frexp(v)[1].max() if v.size else -2139062144   # the fill of 0x80 bytes
        assert scales[k] == want
