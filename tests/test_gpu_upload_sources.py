"""Uploads that return before the copy has run: the copy's host source has to outlive the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


SIZES = [("float64", 1), ("float64", 125), ("float64", 126), ("float64", 4000), ("float64", 4001), ("float32", 100),
         ("float32", 8000), ("int32", 7), ("float64", 0)]   # around one launch and its two argument sizes


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
            assert g.dtype == torch.float64 and g.is_contiguous() and g.data_ptr() % 16 == 0
            assert np.array_equal(g.cpu().numpy(), a)
