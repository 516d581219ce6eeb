"""The parameter sums of the background, in registers for one and two realizations a thread and in shared
memory for more: the same realizations whatever the width."""
import numpy as np
import pytest
import torch

from holodeck_gb300 import cyutils

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nreal", [1, 128, 129, 256, 257, 513])
def test_width_does_not_change_parameter_sums(nreal):
    rng = np.random.default_rng(7)
    nb, nf = 700, 2
    lam = 10.0 ** rng.uniform(-3, 5.5, (nb, 1, 1, nf))
    lam[rng.uniform(size=lam.shape) < 0.3] = 0.0
    lam[::150] = 6e6
    lam = torch.as_tensor(lam, device="cuda")
    h = torch.as_tensor(rng.uniform(1e-31, 1e-29, (nb, 1, 1, nf)), device="cuda")
    grids = [torch.as_tensor(rng.uniform(1.0, 1.9, (nb, 1, 1, nf)), device="cuda") for _ in range(4)]
    order = torch.arange(nb, dtype=torch.int32, device="cuda")
    scales = torch.ones(4, dtype=torch.int32, device="cuda")

    def run(n):
        return cyutils.loudest_par_device(lam, h, n, 2, order, rng_mt, np.ones(1), np.ones(1), grids, scales, seed=3)
    rng_mt = np.linspace(1.0, 2.0, nb) * 1e40
    full, some = run(1000), run(nreal)
    for a, b in zip(full, some):   # (F, R, L), (F, R), (4, F, R, L), (7, F, R)
        axis = 1 if a.shape[0] == nf else 2
        assert torch.equal(b, a.narrow(axis, 0, nreal))
