"""Parameters and images that are views into flat buffers at any offset: the network
copies what its kernels cannot read in place, and the native call refuses it."""
import pytest

pytestmark = pytest.mark.gpu


def flat_views(tensors, offset, dtype):
    """The tensors again, each `offset` elements into a buffer of its own."""
    import torch
    out = []
    for t in tensors:
        flat = torch.zeros(t.numel() + offset, dtype=dtype, device="cuda")
        flat[offset:].copy_(t.detach().reshape(-1))
        out.append(flat[offset:].view(t.shape))
        assert out[-1].is_contiguous()
    return out


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
def test_views_into_flat_buffers(offset):
    import torch
    from langmuir_b200 import surrogate as S
    ph, _, _ = S.grf_morphologies(3, size=128, seed=2)
    x = S.phases_to_input(ph, ramp=0.5)
    params = [p.detach() for p in S.init_params(2)]
    views = flat_views(params, offset, torch.float32)
    assert any(v.data_ptr() % 16 for v in views) == (offset % 4 != 0)
    odd_x, = flat_views([x], offset, torch.bfloat16)
    want, kept = S.network_forward(x, params)
    got, kept_views = S.network_forward(odd_x, views)
    assert torch.equal(got, want)
    dy = torch.ones_like(want)
    # the convolutions' gradients are added by atomics, in any order
    for g, w in zip(S.network_backward(dy, kept_views), S.network_backward(dy, kept)):
        assert torch.linalg.norm(g - w) <= 1e-5 * torch.linalg.norm(w)
    assert S.device_errors() == 0


def test_native_call_refuses_unaligned_buffers():
    import ctypes
    import torch
    from langmuir_b200 import _native as N
    from langmuir_b200 import surrogate as S
    B, H, W = 1, 64, 128
    x = torch.zeros(B * H * W + 2, dtype=torch.bfloat16, device="cuda")
    params = [p.detach() for p in S.init_params(2)]
    views = flat_views(params, 1, torch.float32)
    kept = torch.empty(N.lib().lgm_cnn_net_bytes(B, H, W, 1), dtype=torch.uint8, device="cuda")
    work = torch.empty(N.lib().lgm_cnn_net_bytes(B, H, W, 2), dtype=torch.uint8, device="cuda")
    y = torch.full((B, 2), 7.0, device="cuda")

    def forward(xp, ps):
        ptrs = (ctypes.c_void_p * 12)(*[p.data_ptr() for p in ps])
        return N.lib().lgm_cnn_net_forward(xp, ptrs, kept.data_ptr(), y.data_ptr(), B, H, W, 1,
                                           None)
    INVALID = 1
    for i in (2, 4, 6):
        one = list(params)
        one[i] = views[i]
        assert forward(x.data_ptr(), one) == INVALID
    assert forward(x.data_ptr() + 2, params) == INVALID
    grads = [torch.empty_like(p) for p in params]
    gptrs = (ctypes.c_void_p * 12)(*[g.data_ptr() for g in grads])
    assert N.lib().lgm_cnn_net_backward(x.data_ptr() + 2, kept.data_ptr(), y.data_ptr(),
                                        work.data_ptr(), gptrs, B, H, W, None) == INVALID
    torch.cuda.synchronize()
    assert torch.all(y == 7.0)
    small = list(params)
    for i in (0, 1, 3, 5, 7, 8, 9, 10, 11):  # read word by word
        small[i] = views[i]
    assert forward(x.data_ptr(), small) == N.OK
    torch.cuda.synchronize()
