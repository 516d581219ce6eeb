"""The gradient solve with two and with four lanes a point, either side of the width that picks them: the
density scattered through the phases and one level at a time (rounding is a few ulp a sweep)."""

import pytest

from test_scatter_phases import test_pipelined_solve_matches_level_by_level as _matches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,nz,maxiter", [((56, 20), 3, 400), ((57, 20), 3, 400), ((56, 56), 2, 400),
                                              ((17, 9), 7, 400), ((8, 8), 2, 2), ((64, 33), 2, 400)])
def test_either_side_of_the_rule(built_lib, shape, nz, maxiter):
    _matches(built_lib, shape, nz, maxiter)
