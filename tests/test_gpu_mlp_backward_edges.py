"""The backward pass at the edges of its tiles, bit for bit on small integers: a linear network's weight and
bias gradients with ragged batches (rows beyond the last 128-row split, batches below one), widths that
leave a 64-column tile short, and inputs that do not start on 16 bytes; and the input gradient through
a hidden layer against the oracle."""

import ctypes

import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


def _net(dims, members, rng):
    import torch
    from holodeck_gb300 import emulator as E
    net = E.MLPEnsemble(dims, members=members)
    p = rng.integers(-2, 3, size=(members, net.n_params)).astype(np.float32)
    net.load_params(p)
    return net, p


@pytest.mark.parametrize("k,n,batch,members", [(16, 16, 1, 1), (48, 80, 127, 3), (256, 256, 129, 2), (144, 112, 300, 5),
                                               (16, 240, 640, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_linear_gradients_exact(built_lib, k, n, batch, members, offset):
    import torch
    from holodeck_gb300 import _native as N
    rng = np.random.default_rng(k + n + batch)
    net, p = _net([k, n], members, rng)
    x = rng.integers(-3, 4, size=(batch, k)).astype(np.float32)
    q = rng.integers(-3, 4, size=(batch, n)).astype(np.float32)
    # the outputs that go in are the targets plus q B N / 2, so that d loss / d out is q exactly when
    # B N / 2 is a power of two, and q rounded once (as the oracle rounds it) otherwise
    target = rng.integers(-4, 5, size=(batch, n)).astype(np.float32)
    out = np.broadcast_to(target + q * np.float32(batch * n / 2.0), (members, batch, n)).astype(np.float32)
    want = MO.bf16((np.float32(2.0) / (np.float32(batch) * np.float32(n))) * (out[0] - target))
    flat = torch.zeros(batch * k + 8, dtype=torch.bfloat16, device="cuda")
    flat[offset:offset + batch * k] = torch.as_tensor(x.ravel(), device="cuda").to(torch.bfloat16)
    xt = flat[offset:offset + batch * k]
    act = torch.zeros(16, dtype=torch.bfloat16, device="cuda")
    pre = torch.zeros(16, device="cuda")
    o, t = torch.as_tensor(np.ascontiguousarray(out), device="cuda"), torch.as_tensor(target, device="cuda")
    ws_bytes = N.load().hgb_mlp_backward_workspace_bytes(ctypes.byref(net.struct), batch)
    ws = torch.full((ws_bytes,), 255, dtype=torch.uint8, device="cuda")
    loss = torch.empty(members, device="cuda")
    net.grad.fill_(float("nan"))
    N.call("hgb_mlp_backward", ctypes.byref(net.struct), N.ptr(xt), 0, batch, N.ptr(act), N.ptr(pre), N.ptr(o), N.ptr(t),
           0, N.ptr(net.grad), N.ptr(loss), N.ptr(ws), int(ws_bytes), net.status.ptr, N.stream_handle())
    net.check_status()
    grad = net.grad.cpu().numpy()
    # sums of at most 640 products of bf16 values up to 9: exact in fp32 where want holds integers, a few
    # ulp of the largest partial sum otherwise
    tol = 0.0 if np.array_equal(want, q) else 640 * 9 * 2.0 ** -22
    for m in range(members):
        assert np.all(np.abs(grad[m, :n * k].reshape(n, k) - want.T.astype(np.float64) @ x) <= tol)
        assert np.all(np.abs(grad[m, n * k:] - want.sum(axis=0, dtype=np.float64)) <= tol)
    np.testing.assert_allclose(loss.cpu().numpy(), np.mean((out[0] - target).astype(np.float64) ** 2), rtol=1e-5)


@pytest.mark.parametrize("dims,batch", [([16, 80, 48, 16], 130), ([32, 256, 144, 16], 65)])
def test_hidden_gradients_against_oracle(built_lib, dims, batch):
    import torch
    rng = np.random.default_rng(batch)
    net, _ = _net(dims, 2, rng)
    p = (rng.uniform(-0.3, 0.3, size=(2, net.n_params))).astype(np.float32)
    net.load_params(p)
    x = MO.bf16(rng.uniform(-1, 1, size=(batch, dims[0])).astype(np.float32))
    t = rng.normal(size=(batch, dims[-1])).astype(np.float32)
    loss = net.gradients(torch.as_tensor(x, device="cuda").to(torch.bfloat16),
                         torch.as_tensor(t, device="cuda")).cpu().numpy()
    grad = net.grad.cpu().numpy()
    net.check_status()
    for m in range(2):
        layers = [(MO.bf16(net.layer(p, m, ll)[0]), net.layer(p, m, ll)[1]) for ll in range(len(dims) - 1)]
        exp_loss, grads = MO.backward(layers, x, t)
        assert abs(loss[m] - exp_loss) <= 1e-5 * exp_loss
        off = 0
        for (gw, gb), k, n in zip(grads, dims[:-1], dims[1:]):
            for got, exp in ((grad[m, off:off + n * k].reshape(n, k), gw), (grad[m, off + n * k:off + n * k + n], gb)):
                assert np.linalg.norm(got - exp) <= 2e-3 * np.linalg.norm(exp) + 1e-12
            off += n * k + n
