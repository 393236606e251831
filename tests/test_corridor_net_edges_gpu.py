"""The backward kernels of the corridor CNN at the edges of their tiles: window
sizes around the 16-cell steps, the 32-column form, odd and even heights, one
row, one column and the largest window, with everything outside what the
layout defines poisoned with NaN.

Tolerances.  The head's sums of at most 2 x 63 x 63 f32 products in another
order: relative 1e-3 of the largest element.  Layer 4's weight gradient reads
the head's bf16 gradient, whose elements may differ by a bf16 ulp (2^-8
relative) where the f32 sum of nine products rounds the other way (a few in a
thousand): Frobenius 2^-8 * sqrt(0.005) < 1e-3.  Deeper layers accumulate such
ulps over the convolutions: 1e-2, the bound of the layer-by-layer test.  A
missing or doubled row, column or cell of a window is at least 1/63 of the
cells of a sum, an order above."""

import numpy as np
import pytest
import torch

from apgar_b200 import learned
from oracle import corridor_net as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cw,ch", [(1, 1), (2, 63), (15, 2), (16, 17), (17, 16), (31, 7), (31, 62), (32, 8), (32, 9),
                                   (47, 33), (48, 24), (49, 1), (62, 31), (63, 62), (63, 63), (0, 0)])
def test_gradients_at_the_edges_of_a_tile(cw, ch):
    rng = np.random.default_rng(100 * cw + ch)
    if cw == 0:  # a batch of every kind, more tiles than one pass of the chip
        sizes = [(int(rng.integers(1, 64)), int(rng.integers(1, 64))) for _ in range(24)]
    else:
        sizes = [(cw, ch)] * 2
    n = len(sizes)
    dims = np.array([w | (h << 8) | (2 << 16) for w, h in sizes], np.uint32)
    mask = ref.valid_mask(dims)
    x0 = np.where(mask[..., None], ref.bf16(rng.random((n, 64, 64, 16)).astype(np.float32)), 0.0)
    padded = np.full((n, 66, 64, 16), np.nan, np.float32)
    for i, (w, h) in enumerate(sizes):
        padded[i, 0:h + 2] = 0.0  # the rows the layout defines
        padded[i, 1:h + 2] = x0[i, 0:h + 1]
    labels = (rng.random((n, 64, 64)) < 0.2).astype(np.uint8)

    net = learned.CorridorNet(seed=7)
    r = torch.from_numpy(padded).cuda().to(torch.bfloat16)
    d = torch.from_numpy(dims.view(np.int32)).cuda()
    acts = net.activations(n, distinct=True)
    for a in acts:
        a.fill_(float("nan"))
    poison = [torch.full_like(acts[0], float("nan")) for _ in range(2)]
    del poison  # the gradient buffers come from here
    logits = net.forward(r, d, acts=acts)
    net.backward(r, d, acts, logits, torch.from_numpy(labels).cuda(), pos_weight=8.0)
    torch.cuda.synchronize()
    net.check_error()

    params = net.params.cpu().numpy()
    grid = lambda a: np.where(mask[..., None], a.float().cpu().numpy()[:, 1:65], 0.0)  # noqa: E731
    x = [x0] + [grid(a) for a in acts]
    z = np.where(mask, logits.cpu().numpy(), 0.0)
    _, dlogit = ref.loss_grad(z, labels, mask, 8.0)
    grads = ref.unflatten(net.grads.cpu().numpy())
    dpre, dw6, db6 = ref.head_backward(x[5], params, dlogit, mask)
    for got, want in ((grads["w6"], dw6), (grads["b6"], db6)):
        assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    for layer in range(4, -1, -1):
        dw, db = ref.weight_grad(x[layer], dpre, mask)
        for got, want in ((grads[f"w{layer}"], dw), (grads[f"b{layer}"], db)):
            err = np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-12)
            assert err < (1e-3 if layer == 4 else 1e-2), (layer, err)
        if layer > 0:
            dpre = ref.input_grad(dpre, params, layer, x[layer], mask)
