"""Background realizations over the block widths (one to eight realizations a thread) and the batches of
inversion tables: every draw is keyed by bin and realization, so neither may show in the results."""
import numpy as np
import pytest
import torch

from holodeck_gb300 import cyutils

pytestmark = pytest.mark.gpu

# expectations at the ends of the table range and where a table changes its cut (2048 entries: lambda
# near 21200; 512: near 1286), with a few of the other kinds between
EDGES = [0.0, 0.05, 9.99, 10.0, 10.01, 25.0, 1280.0, 1286.0, 1292.0, 21100.0, 21190.0, 21300.0, 46999.0, 47000.0,
         47001.0, 3.0]


def _grid(nb, nf, seed):
    rng = np.random.default_rng(seed)
    lam = np.exp(rng.uniform(np.log(10.0), np.log(47000.0), (nb, nf)))
    where = rng.uniform(size=(nb, nf)) < 0.5
    lam[where] = rng.choice(EDGES, size=(nb, nf))[where]
    return lam


@pytest.mark.parametrize("nreal", [1, 127, 128, 129, 256, 257, 512, 513, 1000])
def test_width_does_not_change_realizations(nreal):
    lam = torch.as_tensor(_grid(1500, 3, 1), device="cuda")
    h = torch.as_tensor(np.random.default_rng(2).uniform(1e-30, 1e-28, (1500, 3)), device="cuda")
    order = torch.arange(1500, dtype=torch.int32, device="cuda")
    full = cyutils.sam_poisson_gwb(lam, h, 1024, seed=11)
    assert torch.equal(cyutils.sam_poisson_gwb(lam, h, nreal, seed=11), full[:, :nreal])
    ss, bg = cyutils.loudest_device(lam, h, 1024, 2, order, seed=12)
    ss_n, bg_n = cyutils.loudest_device(lam, h, nreal, 2, order, seed=12)
    assert torch.equal(ss_n, ss[:, :nreal]) and torch.equal(bg_n, bg[:, :nreal])


@pytest.mark.parametrize("nreal", [100, 200, 400, 1000])
def test_tables_do_not_depend_on_their_batch(nreal):
    """With unit strain the sums are counts below 2^24, exact in FP32 in any order: the bins drawn together
    are the sum of the bins drawn a few at a time."""
    nb = 128
    lam = _grid(nb, 2, 3)
    lam[lam < 10.0] = 0.0   # (the other kinds' sums are not all integers below 2^24 of the same unit)
    lam[lam > 47000.0] = 0.0
    assert lam.sum(axis=0).max() * 1.1 < 2 ** 24
    one = torch.ones((nb, 2), dtype=torch.float64, device="cuda")
    draw = lambda x: cyutils.sam_poisson_gwb(torch.as_tensor(x, device="cuda"), one, nreal, seed=4)
    total = draw(lam)
    parts = torch.zeros_like(total)
    for k in range(16):
        some = lam.copy()
        some[np.arange(nb) % 16 != k] = 0.0
        parts += draw(some)
    assert torch.equal(total, parts)
    assert float(total.max()) < 2 ** 24


@pytest.mark.parametrize("lam", [10.0, 56.0, 1286.0, 21190.0, 21300.0, 47000.0])
def test_table_moments(lam):
    """Mean and variance of the drawn counts within six of their standard deviations."""
    nr = 20000
    n = cyutils.sam_poisson_gwb(torch.full((1, 1), lam, dtype=torch.float64, device="cuda"),
                                torch.ones((1, 1), dtype=torch.float64, device="cuda"), nr, seed=8).cpu().numpy()[0]
    assert np.array_equal(n, np.rint(n))
    assert abs(n.mean() - lam) < 6 * np.sqrt(lam / nr)
    assert abs(n.var() - lam) < 6 * lam * np.sqrt((2 + 1 / lam) / nr)
