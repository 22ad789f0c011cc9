"""Layer 4's weight gradient beside the end of the image: what lies in the image's last row
does not reach the taps that would meet it only past the image."""
import math

import pytest
import torch

from langmuir_b200 import surrogate as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [64, 128, 192])  # layer 4: 8, 16 and 24 rows, in tiles of 16
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_rows_past_the_image_add_nothing(H, value):
    B, W = 3, 128
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(B, H, W, 1, generator=g, device="cuda").to(torch.bfloat16)
    params = [p.detach() for p in S.init_params(3)]
    dy = torch.randn(B, 2, generator=g, device="cuda")
    _, saved = S.network_forward(x, params)
    want = S.network_backward(dy, saved)[6].view(32, 3, 3, 32)
    # layer 4's inputs in what the forward call kept: planes [B][4][H/8][W/8][8] behind the
    # first two layers' outputs
    at = B * H * W * (16 + 4)
    p3 = saved[1][at:at + B * H * W].view(torch.bfloat16).view(B, 4, H // 8, W // 8, 8)
    p3[1, :, -1] = value
    got = S.network_backward(dy, saved)[6].view(32, 3, 3, 32)
    assert not torch.isfinite(got[:, 1:]).any()  # every tap that sees the row, in the image
    # the first row of taps sees the last row of inputs only past the image: the same FP32
    # sums, up to the order in which the CTAs add theirs
    assert torch.isfinite(got[:, 0]).all()
    assert (got[:, 0] - want[:, 0]).norm() <= 1e-5 * want[:, 0].norm()
