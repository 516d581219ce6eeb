"""The hardening normalisation against the oracle where a warp's cells and a lane's steps run out: cell
counts off a multiple of the cells per warp and either side of the rule that picks it, steps off a
multiple of the lanes' share, the largest count held in registers and the first beyond it, planned and
general exponents, and times that no normalisation reaches."""

import numpy as np
import pytest

from oracle import sam_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,gi,go,time", [
    (1, 300, -1.0, 2.5, 3.0), (3, 1, -1.0, 2.5, 3.0), (5, 7, -0.5, 2.5, 1.0), (2431, 40, -1.0, 2.5, 3.0),
    (2433, 41, 0.0, 1.5, 3.0), (9, 319, -0.7, 2.5, 0.5), (6, 320, -1.0, 3.0, 3.0), (6, 321, -1.0, 3.0, 3.0),
    (7, 300, -1.0, 2.5, 1e-30)])
def test_norm_at_the_edges(built_lib, n, steps, gi, go, time):
    from holodeck_gb300 import constants as C
    from holodeck_gb300.sams import sam_cyutils
    rng = np.random.default_rng(n + steps)
    mt, mr = 10.0 ** rng.uniform(4, 12, n) * C.MSOL, 10.0 ** rng.uniform(-3, 0, n)
    args = (time * C.GYR, mt, mr, 1e3 * C.PC, 100.0 * C.PC, gi, go, steps)
    want = np.zeros(n)
    for ii in range(n):   # scipy's Python brentq raises where its Cython one, and the kernel, give 0
        try:
            want[ii] = O.find_2pwl_hardening_norm(args[0], mt[ii:ii + 1], mr[ii:ii + 1], *args[3:])[0]
        except ValueError:
            pass
    got, norm = sam_cyutils.find_2pwl_hardening_norm(*args, return_norm=True)
    # the root is known to 1e-3; iterates follow the reference's to the lifetime's rounding, 1e-13 at most
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-10)
    np.testing.assert_allclose(norm, 10.0 ** want, rtol=1e-9)
