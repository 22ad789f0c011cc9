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


@pytest.mark.parametrize("n,H,W,seed", [(256, 128, 128, 1), (256, 128, 128, 2), (33, 64, 256, 3),
                                        (1, 64, 128, 4)])
def test_native_forward_has_the_layers_bits(n, H, W, seed):
    """The native forward pass adds in the per-layer kernels' order, so no BF16
    activation rounds the other way: the outputs are equal, not close."""
    import torch
    from langmuir_b200 import surrogate as S
    ph, _, _ = S.grf_morphologies(n, size=max(H, W), seed=seed)
    x = S.phases_to_input(ph[:, :H, :W].contiguous(), ramp=0.5)
    params = S.init_params(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for i in (1, 3, 5, 7, 9, 11):
            params[i].copy_(torch.randn(params[i].shape, generator=g, device="cuda") * 0.1)
        y, _ = S.network_forward(x, params, keep=False)
        c1w, c1b, c2w, c2b, c3w, c3b, c4w, c4b, f1w, f1b, f2w, f2b = params
        p = x
        for k, (w, b, cin) in enumerate([(c1w, c1b, 1), (c2w, c2b, S.CH), (c3w, c3b, S.CH)]):
            _, p = S.conv3x3(p, S.conv_weights_bf16(w, cin), b, H >> k, W >> k, keep_act=False)
        a4, _ = S.conv3x3(p, S.conv_weights_bf16(c4w, S.CH), c4b, H >> 3, W >> 3, pool=False)
        _, g16 = S.gap_fwd(a4)
        hid, out = S.HIDDEN, S.OUTPUTS
        h = S.to_bf16(S.gemm(g16, S.CH, 1, f1w.to(torch.bfloat16), 1, S.CH, n, hid, S.CH, bias=f1b,
                             relu=True))
        want = S.gemm(h, hid, 1, f2w.to(torch.bfloat16), 1, hid, n, out, hid, bias=f2b)
    np.testing.assert_array_equal(y.cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_non_finite_pixels_reach_their_neighbours_only(value):
    """An infinity or NaN in an image does to its 3x3 neighbourhood what it does in
    the per-layer kernels, and nothing to the pixels beside it."""
    import torch
    from langmuir_b200 import surrogate as S
    H, W = 64, 128
    at = [(0, 0), (5, 2), (5, 3), (10, 16), (10, 31), (11, 32), (20, 63), (33, 64), (63, 127),
          (62, 126), (40, 127), (40, 1)]
    x = S.phases_to_input(torch.zeros(len(at), H, W, dtype=torch.uint8), ramp=0.5)
    for b, (r, c) in enumerate(at):
        x[b, r, c] = value
    params = [p.detach() for p in S.init_params(7)]
    params[1].fill_(0.25)
    y, (_, kept) = S.network_forward(x, params)
    _, p1 = S.conv3x3(x, S.conv_weights_bf16(params[0], 1), params[1], H, W, keep_act=False)
    # layer 1's pooled output, planes of eight channels, comes first in what is kept
    planes = kept[:p1.numel() * 2].view(torch.bfloat16).view(len(at), 4, H // 2, W // 2, 8)
    got = planes.permute(0, 2, 3, 1, 4).reshape(p1.shape)
    np.testing.assert_array_equal(got.float().cpu().numpy(), p1.float().cpu().numpy())
