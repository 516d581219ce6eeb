"""The cumulative expectation that the loudest slots are drawn from: an occupied bin is found wherever it
lies among empty ones, at the edges of segments, passes, warps and threads of the scan."""
import numpy as np
import pytest
import torch

from holodeck_gb300 import cyutils

pytestmark = pytest.mark.gpu

SEGMENTS = 64


@pytest.mark.parametrize("nb", [1, 63, 65, SEGMENTS * 128, SEGMENTS * 128 + 1, SEGMENTS * 4096 + 1, SEGMENTS * 9000])
def test_loudest_come_from_the_occupied_bin(nb):
    seg = -(-nb // SEGMENTS)
    places = {0, nb - 1, nb // 2} | {k + d for k in (seg, 4 * seg, 63 * seg) for d in (-1, 0, 3, 4, 127, 128, 4095, 4096)}
    places = sorted(p for p in places if 0 <= p < nb)
    nf = len(places)
    h = np.repeat(np.linspace(2.0, 1.0, nb)[:, None], nf, axis=1) * 1e-30
    lam = np.zeros((nb, nf))
    lam[:: max(1, nb // 50)] = np.nan     # NaN and negative expectations count as none
    lam[1:: max(1, nb // 40)] = -3.0
    for f, p in enumerate(places):
        lam[p, f] = 500.0   # fewer than three sources have a probability below 1e-200
    ss, _ = cyutils.loudest_device(torch.as_tensor(lam, device="cuda"), torch.as_tensor(h, device="cuda"), 7, 3,
                                   torch.arange(nb, dtype=torch.int32, device="cuda"), seed=5)
    want = np.array([h[p, f] for f, p in enumerate(places)])
    assert np.array_equal(ss.cpu().numpy(), np.broadcast_to(want[:, None, None], (nf, 7, 3)))


@pytest.mark.parametrize("nb", [130, SEGMENTS * 200])
def test_cut_does_not_show(nb):
    """A few thin bins among empty ones: the number of loud sources follows the summed expectation."""
    nr, nl = 4000, 4
    lam = np.zeros((nb, 1))
    where = np.linspace(0, nb - 1, 37).astype(int)
    lam[where, 0] = 0.03   # in all 1.11
    h = np.linspace(2.0, 1.0, nb)[:, None] * 1e-30
    ss, _ = cyutils.loudest_device(torch.as_tensor(lam, device="cuda"), torch.as_tensor(h, device="cuda"), nr, nl,
                                   torch.arange(nb, dtype=torch.int32, device="cuda"), seed=6)
    ss = ss.cpu().numpy()[0]
    assert np.isin(ss[ss > 0], h[where, 0]).all()
    total = lam.sum()
    pk = np.exp(-total) * total ** np.arange(nl) / np.array([1, 1, 2, 6])
    for k in range(nl):   # exactly k sources, within six standard deviations
        n = np.sum((ss > 0).sum(axis=1) == k)
        assert abs(n - nr * pk[k]) < 6 * np.sqrt(nr * pk[k] * (1 - pk[k]))
