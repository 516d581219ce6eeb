"""Uploads that return before the copy has run: the copy's host source has to outlive the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


SIZES = [("float64", 1), ("float64", 125), ("float64", 126), ("float64", 500), ("float64", 501), ("float64", 4000), ("float64", 4001), ("float32", 100),
         ("float32", 8000), ("int32", 7), ("float64", 0)]   # around one launch and its argument sizes


@pytest.mark.parametrize("dtype,n", SIZES)
def test_unawaited_copies_read_pinned_memory(dtype, n):
    import torch
    from torch.utils._python_dispatch import TorchDispatchMode
    from holodeck_gb300 import _device as D

    class Spy(TorchDispatchMode):
        seen = []   # (source is pinned) of every copy from the host that does not wait

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            kwargs = kwargs or {}
            name = func.overloadpacket.__name__
            src = args[0] if name == "_to_copy" else args[1] if name == "copy_" else None
            unawaited = kwargs.get("non_blocking", False) or (name == "copy_" and len(args) > 2 and args[2])
            if src is not None and unawaited and src.device.type == "cpu":
                self.seen.append(src.is_pinned())
            return func(*args, **kwargs)

    host = (np.arange(n) * 1.25).astype(dtype)
    with Spy() as spy:
        got = D.as_device(host, dtype=getattr(torch, dtype))
    assert all(spy.seen)
    assert got.dtype == getattr(torch, dtype) and tuple(got.shape) == (n,)
    assert np.array_equal(got.cpu().numpy(), host)


def test_many_uploads_behind_queued_work():
    """Freed host blocks of the same size are filled with other values while the uploads wait."""
    import torch
    from holodeck_gb300 import _device as D
    big = torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    for _ in range(10):
        big.add_(1.0)
    got, fill = [], []
    for k in range(300):
        n = 1 + 13 * (k % 300)
        got.append((k, n, D.as_device(np.full(n, float(k)))))
        fill.append(np.full(n, -1.0))
        if k % 3 == 0:
            fill.clear()
    for k, n, x in got:
        assert torch.equal(x.cpu(), torch.full((n,), float(k), dtype=torch.float64)), k


def test_arrays_that_travel_together():
    import torch
    from holodeck_gb300 import _device as D
    host = [np.arange(5.0), np.linspace(0.0, 1.0, 8)[::2], np.array([[1.5, 2.5], [3.5, 4.5]])]
    tensor = torch.arange(3.0, dtype=torch.float64, device="cuda")
    for arrs in (host, host[:1], [host[0], tensor, host[1]], [np.arange(4), host[0]], [np.empty(0), host[0]],
                 [np.arange(3000.0), np.arange(3001.0)]):
        got = D.as_devices(*arrs)
        for g, a in zip(got, arrs):
            a = a.cpu().numpy() if a is tensor else a
            assert g.dtype == torch.float64 and g.is_contiguous() and g.data_ptr() % 8 == 0
            assert np.array_equal(g.cpu().numpy(), a)


def test_batch_work_list_outlives_the_call(built_lib):
    """A captured multi-sample launch replays from its own copy of the work list, whatever the host memory that
    the call built it in holds by then (lists of one and of several uploads)."""
    import torch
    from holodeck_gb300 import _device as D, cyutils, single_sources
    rng = np.random.default_rng(3)
    for nf, sizes in ((2, ((300, 5),)), (40, ((9000, 60), (7000, 1100)))):
        samples = []
        for nb, nr in sizes:
            num, hh = (torch.as_tensor(10.0 ** rng.uniform(lo, hi, size=(nb, nf)), device="cuda")
                       for lo, hi in ((-4.0, 6.0), (-32.0, -26.0)))
            samples.append(dict(number=num, h2fdf=hh, order=single_sources.sort_order_device(hh), nreals=nr, seed=nb,
                                status=D.StatusWord()))
        want = cyutils.loudest_batch_device(samples, 3)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            got = cyutils.loudest_batch_device(samples, 3)
        fill = [np.full(1 << k, 0xFFFFFFFF, dtype=np.uint32) for k in range(4, 18) for _ in range(8)]
        for _ in range(2):
            for ss, bg in got:
                ss.fill_(-1.0)
                bg.fill_(-1.0)
            graph.replay()
            torch.cuda.synchronize()
            for (ss, bg), (want_ss, want_bg) in zip(got, want):
                assert torch.equal(ss, want_ss) and torch.equal(bg, want_bg)
        del fill
