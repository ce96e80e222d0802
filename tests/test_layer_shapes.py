"""Input shapes of the layer: a matrix is taken as it is, everything else is reshaped. Runs without a GPU."""
import pytest
import torch

from ccfuser_b200 import MoEConfig, MoELayer


@pytest.fixture
def layer():
    torch.manual_seed(0)
    return MoELayer(MoEConfig(d_model=64, d_ffn=128, num_experts=4, top_k=2, activation="gelu", dtype=torch.float32, backend="cpu",
                              max_tokens=12))


@pytest.mark.parametrize("shape", [(12, 64), (3, 4, 64), (2, 2, 3, 64)])
def test_outputs_have_the_shape_of_the_input(layer, shape):
    x = torch.randn(12, 64)
    want = layer(x)
    a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    got = layer(a.view(shape))
    assert got.shape == shape and torch.equal(got.reshape(12, 64), want)
    got.sum().backward()
    layer(b).sum().backward()
    assert torch.equal(a.grad, b.grad)


def test_rows_that_are_not_tokens_are_refused(layer):
    with pytest.raises(RuntimeError):
        layer(torch.randn(24, 32))     # two rows to a token: the output cannot have this shape


def test_a_matrix_with_other_strides(layer):
    x = torch.randn(64, 12).t()
    assert torch.equal(layer(x), layer(x.contiguous()))
