"""A density whose kernels may be in flight is not on the model, where another thread would find it and read it
on its own stream; once the call returns it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_density_appears_when_it_is_checked(built_lib, monkeypatch):
    import holodeck_gb300 as H
    from holodeck_gb300 import constants as C, hardening, utils
    from holodeck_gb300.sams import sam as S, sam_cyutils
    model = S.Semi_Analytic_Model(shape=(14, 11, 9), gpf=H.sams.GPF_Power_Law(), gmt=H.sams.GMT_Power_Law())
    model._mmbulge._scatter_dex = 0.3
    hard = hardening.Fixed_Time_2PL_SAM(model, 3.0 * C.GYR)
    seen = []
    run = sam_cyutils.dbn_2pwl_device

    def watched(*args, **kwargs):
        out = run(*args, **kwargs)
        seen.append(model._density_t is None and model._gmt_time_t is None and model._redz_prime_t is None)
        return out

    monkeypatch.setattr(sam_cyutils, "dbn_2pwl_device", watched)
    edges = utils.pta_freqs(16.0 * C.YR, 4)[1]
    first = model.gwb(edges, hard=hard, realize=5, loudest=2, seed=1)
    assert len(seen) == 2 and all(seen)   # the walk beside the scatter, and the evaluation after it
    assert model._density_t is not None and model._gmt_time_t is not None and model._redz_prime_t is not None
    again = model.gwb(edges, hard=hard, realize=5, loudest=2, seed=1)
    for a, b in zip(first, again):
        assert np.array_equal(a, b)


def test_a_check_that_raises_keeps_nothing(built_lib, monkeypatch):
    """The scatter beside the walk (a model with merger times), stopped after one sweep."""
    import functools
    import warnings

    import holodeck_gb300 as H
    from holodeck_gb300 import constants as C, hardening, utils
    from holodeck_gb300.sams import sam as S, scatter
    monkeypatch.setattr(scatter, "add_scatter_to_masses_device",
                        functools.partial(scatter.add_scatter_to_masses_device, maxiter=1))
    edges = utils.pta_freqs(16.0 * C.YR, 4)[1]
    model = S.Semi_Analytic_Model(shape=(14, 11, 9), gpf=H.sams.GPF_Power_Law(), gmt=H.sams.GMT_Power_Law())
    model._mmbulge._scatter_dex = 0.3
    hard = hardening.Fixed_Time_2PL_SAM(model, 3.0 * C.GYR)
    for _ in range(2):   # a second call solves, and raises, again
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            with pytest.raises(UserWarning, match="did not converge"):
                model.gwb(edges, hard=hard, realize=5, loudest=2, seed=1)
        assert model._density_t is None and model._gmt_time_t is None
    with pytest.warns(UserWarning, match="did not converge"):
        model.gwb(edges, hard=hard, realize=5, loudest=2, seed=1)
    assert model._density_t is not None
