"""The hardening normalisation's nodes, shared by a block's cells of one total mass: the same bits however
the cells are ordered, and so however many masses a block meets."""

import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,run,steps,gi", [(8, 8, 300, -1.0), (9, 3, 300, -0.7), (16, 5, 129, -1.0), (17, 17, 128, 0.5),
                                            (1216, 81, 300, -1.0), (1217, 81, 320, -0.7), (1300, 7, 300, -1.0)])
def test_order_does_not_show(built_lib, n, run, steps, gi):
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam_cyutils
    rng = np.random.default_rng(n)
    mt = np.repeat(10.0 ** rng.uniform(4, 12, -(-n // run)) * C.MSOL, run)[:n]
    mr = 10.0 ** rng.uniform(-3, 0, n)
    rest = (1e3 * C.PC, 100.0 * C.PC, gi, 2.5, steps)
    got = sam_cyutils.find_2pwl_hardening_norm(3.0 * C.GYR, mt, mr, *rest)
    perm = rng.permutation(n)
    assert np.array_equal(sam_cyutils.find_2pwl_hardening_norm(3.0 * C.GYR, mt[perm], mr[perm], *rest), got[perm])
    some = perm[:8]   # against the oracle (the lifetime's rounding, as in the edge tests)
    want = O.find_2pwl_hardening_norm(3.0 * C.GYR, mt[some], mr[some], *rest)
    np.testing.assert_allclose(got[some], want, rtol=0, atol=1e-10)
