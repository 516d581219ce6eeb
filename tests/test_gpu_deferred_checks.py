"""Status words that are read after the last launch: what a stage reports still reaches the caller, in stage
order, and a density whose check failed is not kept."""
import functools
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model():
    from holodeck_gb300 import hardening
    from holodeck_gb300.sams import sam as S
    model = S.Semi_Analytic_Model(shape=(14, 11, 9))
    model._mmbulge._scatter_dex = 0.3
    hard = hardening.Fixed_Time_2PL_SAM(model, 3.0)
    return model, hard


def _edges(nf=4):
    from holodeck_gb300 import utils, constants as C
    return utils.pta_freqs(16.0 * C.YR, nf)[1]


@pytest.fixture
def one_sweep(monkeypatch):
    from holodeck_gb300.sams import scatter
    monkeypatch.setattr(scatter, "add_scatter_to_masses_device",
                        functools.partial(scatter.add_scatter_to_masses_device, maxiter=1))


def test_unconverged_gradients_warn(built_lib, one_sweep):
    model, hard = _model()
    with pytest.warns(UserWarning, match="did not converge"):
        model.gwb(_edges(), hard=hard, realize=5, loudest=2, seed=1)
    assert model._density_t is not None


def test_a_warning_that_raises_keeps_no_density(built_lib, one_sweep):
    model, hard = _model()
    for _ in range(2):   # a second call solves, and raises, again
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            with pytest.raises(UserWarning, match="did not converge"):
                model.gwb(_edges(), hard=hard, realize=5, loudest=2, seed=1)
        assert model._density_t is None


def test_stage_order_of_failures(built_lib, one_sweep):
    """A refused replay comes after the scatter's warning, as when every stage was checked in turn."""
    model, hard = _model()
    with pytest.warns(UserWarning, match="did not converge"):
        with pytest.raises(ValueError, match="replay must be shaped"):
            model.gwb(_edges(), hard=hard, realize=5, loudest=2, seed=1, replay=np.zeros((1, 1, 1)))


@pytest.mark.parametrize("n", [1, 4096, 4097, 20000])
def test_uploads_hold_the_values_of_the_call(n):
    """An upload that does not wait: the array may change as soon as the call returns."""
    import torch
    from holodeck_gb300 import _device as D
    big = torch.zeros(1 << 26, device="cuda")
    arr = np.arange(n, dtype=np.float64)
    for _ in range(3):
        big.add_(1.0)   # work that the stream still has before it
    got = D.as_device(arr)
    arr[:] = -1.0
    assert torch.equal(got.cpu(), torch.arange(n, dtype=torch.float64))


def test_kept_edges_are_there_for_other_streams(built_lib):
    """A model's edges are read on another stream than the one whose queue was busy when they were made."""
    import torch
    from holodeck_gb300.sams import sam as S
    model = S.Semi_Analytic_Model(shape=(14, 11, 9))
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    big = torch.zeros(1 << 27, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        for _ in range(20):
            big.add_(1.0)
        edges = model._edges_device()
    with torch.cuda.stream(other):
        got = [e.clone() for e in edges]
        other.synchronize()
    for g, want in zip(got, model.edges):
        assert np.array_equal(g.cpu().numpy(), np.asarray(want, dtype=np.float64))


def test_uploads_are_refused_under_capture():
    import torch
    from holodeck_gb300 import _device as D
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(graph):
            D.as_device(np.arange(4.0))
    torch.cuda.synchronize()
