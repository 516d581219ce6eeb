"""Bins of 2^22 sources and more, which the chunks take in runs of four: every one is drawn once, whatever
the number of bins.  With unit strain the sums are whole numbers, exact in FP64 in any order."""
import numpy as np
import pytest
import torch

from holodeck_gb300 import cyutils

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 3, 4, 5, 127, 129, 1025, 3001])
@pytest.mark.parametrize("nreal", [3, 200])
def test_each_wide_bin_once(nb, nreal):
    rng = np.random.default_rng(nb)
    lam = rng.uniform(4.2e6, 9e6, (nb, 2))
    one = torch.ones((nb, 2), dtype=torch.float64, device="cuda")
    draw = lambda x: cyutils.sam_poisson_gwb(torch.as_tensor(x, device="cuda"), one, nreal, seed=9)
    total = draw(lam)
    parts = torch.zeros_like(total)
    for k in range(3):
        some = lam.copy()
        some[np.arange(nb) % 3 != k] = 0.0
        parts += draw(some)
    assert torch.equal(total, parts)
    want = lam.sum(axis=0)[:, None]
    assert np.all(np.abs(total.cpu().numpy() - want) < 8 * np.sqrt(want))
    order = torch.arange(nb, dtype=torch.int32, device="cuda")
    ss, bg = cyutils.loudest_device(torch.as_tensor(lam, device="cuda"), one, nreal, 2, order, seed=9)
    loud = bg.cpu().numpy() + ss.cpu().numpy().sum(axis=-1)
    assert np.all(np.abs(loud - want) < 8 * np.sqrt(want))
