"""The network's two native calls against the FP64 oracle at the edges of their
tiles: images 16 or 8 rows high at layer 4, one image, odd batches, wide ones."""
import zlib

import numpy as np
import pytest

from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 64, 128), (3, 64, 256), (2, 128, 128), (5, 192, 128),
                                   (1, 64, 384)])
def test_native_network_matches_oracle(B, H, W):
    """Forward and backward against the FP64 oracle with the kernels' BF16
    rounding points (1e-2 of each tensor's norm: BF16 keeps 8 bits, and a sum in
    another order moves a value to the next one at most)."""
    import torch
    from langmuir_b200 import surrogate as S
    rng = np.random.default_rng(zlib.crc32(f"net{B}{H}{W}".encode()))
    ph = (rng.random((B, H, W)) < 0.5).astype(np.uint8)
    P = [p.astype(np.float32) for p in C.init_params(3)]
    for i in (1, 3, 5, 7, 9, 11):
        P[i] = (rng.standard_normal(P[i].shape) * 0.1).astype(np.float32)
    params = [torch.as_tensor(p).cuda().requires_grad_(True) for p in P]
    y = S.SurrogateFn.apply(S.phases_to_input(ph), *params)
    R = rng.standard_normal(y.shape)
    loss = (y * torch.as_tensor(R, dtype=torch.float32).cuda()).sum()
    with torch.no_grad():  # the backward pass reads the weights of the forward pass
        for p in params:
            p.add_(1.0)
    loss.backward()
    torch.cuda.synchronize()
    assert S.device_errors() == 0
    y_ref, cache = C.forward(ph, [p.astype(np.float64) for p in P], bf16=True)
    g_ref = C.backward(R, cache, bf16=True)
    yg = y.detach().cpu().numpy()
    assert np.linalg.norm(yg - y_ref) <= 1e-2 * np.linalg.norm(y_ref)
    for (name, shape), p, gr in zip(S.PARAM_SHAPES, params, g_ref):
        g = p.grad.cpu().numpy().astype(np.float64)
        assert g.shape == shape
        assert np.linalg.norm(g - gr) <= 1e-2 * np.linalg.norm(gr), name
    with torch.no_grad():
        again, _ = S.network_forward(S.phases_to_input(ph),
                                     [torch.as_tensor(p).cuda() for p in P], keep=False)
    np.testing.assert_array_equal(again.cpu().numpy(), yg)
