"""The warm start's sliced weight gradients and fused ReLU at the sizes where they change.

Rows around one slice (256), a whole number of slices and the cap (32 slices),
remainders of the 16-row chunks, and hidden widths that do not fill the 64-wide
tiles.  Against the same network in FP64 with BF16-rounded weights: FP32 sums of
at most 16,400 products of order one, 2e-5 of the largest gradient entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hidden", [(1, 8), (17, 224), (255, 64), (256, 65), (257, 224), (512, 100), (513, 224),
                                         (8192, 40), (8193, 224), (16400, 33)])
def test_gradient_matches_fp64(v2g, rows, hidden):
    import torch

    rng = np.random.default_rng(rows + hidden)
    net = v2g.WarmStart(hidden=hidden)
    dims = [16, hidden, hidden, hidden, 3]
    layers = [(rng.normal(0, (2.0 / i) ** 0.5, (o, i)).astype(np.float32), rng.normal(0, 0.05, o).astype(np.float32))
              for i, o in zip(dims, dims[1:])]
    net.params = np.concatenate([v.reshape(-1) for layer in layers for v in layer])
    f = rng.uniform(-1, 1, (rows, 16)).astype(np.float32)
    t = rng.normal(0, 0.3, (rows, 3)).astype(np.float32)
    loss, grad = net.gradient(f, t)
    ws = [(torch.from_numpy(w).bfloat16().double().requires_grad_(), torch.from_numpy(b).double().requires_grad_())
          for w, b in layers]
    y = torch.from_numpy(f).double()
    for k, (w, b) in enumerate(ws):
        y = y @ w.T + b
        if k < 3:
            y = y.clamp_min(0.0)
    want_out = y.detach().numpy()
    want = (y - torch.from_numpy(t).double()).square().mean()
    want.backward()
    g = np.concatenate([v.grad.numpy().reshape(-1) for layer in ws for v in layer])
    assert np.abs(net.forward(f) - want_out).max() <= 2e-5 * max(1.0, np.abs(want_out).max())
    want = float(want.detach())
    assert abs(loss - want) <= 2e-5 * want
    assert np.abs(grad - g).max() <= 2e-5 * np.abs(g).max()
    # the same call again gives the same bits
    loss2, grad2 = net.gradient(f, t)
    assert loss2 == loss and np.array_equal(grad2, grad)
