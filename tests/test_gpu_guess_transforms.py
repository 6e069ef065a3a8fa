"""The element-wise pieces of the learned guess under what torch does to its
own operations: other types, unaligned slices, forward mode, vmap, tracing.
Each is compared with the torch expression; where that is taken the values are
the same, else they differ by a BF16 step at most."""
import pytest
import torch
import torch.autograd.forward_ad as fw

pytestmark = pytest.mark.gpu


def _x(*shape, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(len(shape) + shape[0])
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


def _mean(x):
    Bn, H, W, Cc = x.shape
    return x.view(Bn, H // 2, 2, W // 2, 2, Cc).float().mean((2, 4)).to(torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_pool_of_other_types(dtype):
    from glide_b200.guess import _pool
    x = _x(1, 6, 10, 16, dtype=dtype)
    assert torch.equal(_pool(x), _mean(x))


def test_pool_of_an_unaligned_slice():
    from glide_b200.guess import _pool
    x = _x(1 + 2 * 6 * 10 * 16)[1:].view(2, 6, 10, 16)
    assert x.data_ptr() % 16 and torch.equal(_pool(x), _mean(x))


def test_pool_in_forward_mode_and_vmap():
    from glide_b200.guess import _pool
    x, t = _x(1, 4, 8, 8), _x(2, 4, 8, 8)[:1]
    with fw.dual_level():
        tan = fw.unpack_dual(_pool(fw.make_dual(x, t))).tangent
        ref = fw.unpack_dual(_mean(fw.make_dual(x, t))).tangent
        assert tan is not None and torch.equal(tan, ref)
    xs = _x(3, 1, 4, 8, 8)
    assert torch.equal(torch.func.vmap(_pool)(xs), torch.func.vmap(_mean)(xs))
