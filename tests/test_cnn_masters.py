"""Shapes of the network's parameters: what the kernels would read past is refused."""
import pytest
import torch

from langmuir_b200 import surrogate as S


def _params():
    g = torch.Generator().manual_seed(0)
    return [torch.randn(shape, generator=g) for _, shape in S.PARAM_SHAPES]


@pytest.mark.parametrize("shape", [(9, 32), (32, 3), (32, 1, 3, 3), (8,)])
def test_first_layer_weights_of_another_shape_are_refused(shape):
    ps = _params()
    ps[0] = torch.zeros(shape)
    with pytest.raises(RuntimeError):
        S.conv_weights_bf16(ps[0], 1)
    with pytest.raises(RuntimeError):
        S._masters(ps)


@pytest.mark.parametrize("shape", [(1, 9), (32, 1), (9,), (), (1, 32, 9)])
def test_first_layer_weights_are_broadcast(shape):
    ps = _params()
    ps[0] = torch.randn(shape)
    got = S._masters(ps)[0][0]
    assert got.shape == (32, 9)
    assert torch.equal(got.to(torch.bfloat16), S.conv_weights_bf16(ps[0], 1)[:, :9])


@pytest.mark.parametrize("i", range(1, 12))
def test_short_parameters_are_refused(i):
    ps = _params()
    ps[i] = ps[i].reshape(-1)[:-1]
    with pytest.raises(ValueError):
        S._masters(ps)


def test_parameters_of_the_network_are_passed_on():
    ps = _params()
    ps[2] = ps[2].view(32, 9, 32)  # the same entries
    got, ptrs = S._masters(ps)
    assert [a.data_ptr() for a in got] == [p.data_ptr() for p in ps] == list(ptrs)
