"""What the projections refuse, by shape and by device, before anything is allocated or launched.

The shapes are looked at ahead of the device, so the same cases run on CPU tensors."""
import pytest
import torch

from inferno_b200 import linear as L

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


def bf16(*shape, device):
    return torch.zeros(shape, dtype=torch.bfloat16, device=device)


# The last axis of x is not in_features, but the number of elements divides by it (16 x 1536 is 32 rows of 768, 16 x 384 is 8) or not.
@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("shape", [(16, 1536), (16, 384), (4, 4, 1536), (2, 100), (768, 16), (12288,), ()])
def test_input_width_must_be_in_features(built_lib, device, shape):
    x, w, b = bf16(*shape, device=device), bf16(768, 2304, device=device), bf16(2304, device=device)
    lin = L.Linear(768, 2304).to(device=device, dtype=torch.bfloat16)
    dy = bf16(*shape[:-1], 2304, device=device)
    for call in (lambda: L.linear_forward(x, w, b), lambda: lin(x), lambda: lin(x.requires_grad_()), lambda: L.linear_backward(x.detach(), w, dy)):
        with pytest.raises(ValueError, match="last axis"):
            call()


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dy_shape", [(16, 48), (8, 64), (32, 64), (16,), ()])
def test_gradient_must_have_the_outputs_shape(built_lib, device, dy_shape):
    x, w = bf16(16, 32, device=device), bf16(32, 64, device=device)
    with pytest.raises(ValueError, match="dy must"):
        L.linear_backward(x, w, bf16(*dy_shape, device=device))


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("n", [0, 8, 63, 128])
def test_bias_must_have_one_element_per_column(built_lib, device, n):
    x, w = bf16(16, 32, device=device), bf16(32, 64, device=device)
    for dt in (torch.bfloat16, torch.float32):
        with pytest.raises(ValueError, match="bias"):
            L.linear_forward(x, w, torch.zeros(n, dtype=dt, device=device))


@pytest.mark.gpu
def test_operands_must_share_a_device():
    x, w, b, dy = bf16(16, 32, device="cuda"), bf16(32, 64, device="cuda"), bf16(64, device="cuda"), bf16(16, 64, device="cuda")
    for call in (lambda: L.linear_forward(x, w, b.cpu()), lambda: L.linear_forward(x, w, b.float().cpu())):
        with pytest.raises(ValueError, match="the bias is on cpu"):
            call()
    for call in (lambda: L.linear_forward(x, w.cpu(), b), lambda: L.linear_backward(x, w.cpu(), dy), lambda: L.linear_backward(x, w, dy.cpu())):
        with pytest.raises(RuntimeError, match="not on a CUDA device"):
            call()
    with pytest.raises(ValueError):
        L.linear_forward(x, w[0], b)
