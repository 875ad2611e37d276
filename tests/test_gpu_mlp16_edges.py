"""The warm-start network's kernels at the edges of their tiles (64 x 64
products, 256-row column sums, 8-row loss blocks): loss and gradient against
64 bits on the same BF16-rounded weights."""
import numpy as np
import pytest
import torch

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1), (63, 65, 1), (64, 64, 64), (65, 33, 130)])
@pytest.mark.parametrize("n", [1, 8, 255, 257, 600])
def test_gradient(n, dims):
    rng = np.random.default_rng(n + sum(dims))
    layers = [((rng.normal(size=(a, b)) / np.sqrt(a)).astype(np.float32), rng.normal(size=b).astype(np.float32))
              for a, b in zip(dims[:-1], dims[1:])]
    x = rng.normal(size=(n, dims[0])).astype(np.float32)
    y = rng.normal(size=(n, dims[-1])).astype(np.float32)
    rows = (np.arange(n) % 3 != 1).astype(np.uint8)
    loss, grad = native.mlp16_grad(layers, x, y, rows)
    p = [torch.tensor(a).bfloat16().double().requires_grad_(True) if a.ndim == 2
         else torch.tensor(a).double().requires_grad_(True) for w in layers for a in w]
    h = torch.tensor(x).double()
    for i in range(0, len(p), 2):
        h = h @ p[i] + p[i + 1]
        h = torch.tanh(h) if i + 2 < len(p) else h
    keep = torch.tensor(rows).double()[:, None]
    ref = ((h - torch.tensor(y).double()) ** 2 * keep).sum() / (keep.sum() * dims[-1])
    ref.backward()
    # FP32 sums of up to 600 terms in order: n eps / 2 of the terms' absolute sum; activations carry a few eps
    assert abs(loss - float(ref)) < 1e-4 * float(ref)
    for (dw, db), i in zip(grad, range(0, len(p), 2)):
        for got, want in ((dw, p[i].grad.numpy()), (db, p[i + 1].grad.numpy())):
            assert np.linalg.norm(got - want) < 1e-4 * np.linalg.norm(want) + 1e-7
