"""The gradient solve of a grid beyond shared memory, with fewer slices than multiprocessors (a block each)
and with more (two blocks a multiprocessor): a slice's result does not depend on the others."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [1, 2, 150])
def test_slices_do_not_depend_on_their_number(built_lib, more):
    import torch
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import scatter as S
    nm, nq = 171, 91   # 15561 points: 249 KB of gradients a slice
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mtot = np.logspace(4, 11, nm) * C.MSOL
    mrat = np.logspace(-3, 0, nq)
    rng = np.random.default_rng(4)
    x, y, z = np.linspace(0, 1, nm)[:, None, None], np.linspace(0, 1, nq)[None, :, None], rng.uniform(1, 3, sms + more)
    dens = np.exp(-8.0 * x * z + np.sin(3.0 * y * z)) * rng.uniform(0.9, 1.1, (nm, nq, sms + more))
    full = S.add_scatter_to_masses(mtot, mrat, dens, 0.3)
    few = S.add_scatter_to_masses(mtot, mrat, np.ascontiguousarray(dens[..., :9]), 0.3)
    # (the redistribution sums a row's positive and negative weights over at most 364 nodes; slices are
    # grouped by the count, so allow for a regrouping: 364 x 2^-53 of the largest value of a row)
    assert np.all(np.abs(full[..., :9] - few) <= 4.1e-14 * np.abs(few).max(axis=(0, 1)))
    last = S.add_scatter_to_masses(mtot, mrat, np.ascontiguousarray(dens[..., -3:]), 0.3)
    assert np.all(np.abs(full[..., -3:] - last) <= 4.1e-14 * np.abs(last).max(axis=(0, 1)))
