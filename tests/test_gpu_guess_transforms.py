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


def _fields(n=4, dtype=torch.float32):
    return [_x(n, 6, 10, dtype=dtype).abs() + 0.1 for _ in range(4)]


def _network_input(H, bed, beta, B):
    x = torch.stack([H / 1000.0, bed / 1000.0, (torch.log(torch.clamp(beta, min=1e-8)) + 2.2) / 0.7, B / 35.0], dim=-1)
    return torch.cat([x, torch.zeros(x.shape[:-1] + (4,), device=x.device)], dim=-1).to(torch.bfloat16)


def test_features_in_forward_mode_and_vmap():
    from glide_b200.guess import features
    f = _fields()
    with fw.dual_level():
        d = [fw.make_dual(t, torch.ones_like(t)) for t in f]
        tan = fw.unpack_dual(features(*d)).tangent
        assert tan is not None and torch.equal(tan, fw.unpack_dual(_network_input(*d)).tangent)
    m = [t.unsqueeze(1) for t in f]
    assert torch.equal(torch.func.vmap(features)(*m), torch.func.vmap(_network_input)(*m))


def test_features_are_traced():
    """A traced function follows its inputs."""
    from glide_b200.guess import features
    a, b = _fields(), [t + 1.0 for t in _fields()]
    traced = torch.jit.trace(features, tuple(a), check_trace=False)
    assert torch.equal(traced(*b), _network_input(*b))


def test_faces_of_a_mapped_or_tangent_prediction():
    """The network's output reaches the faces with its tangent."""
    from glide_b200 import guess

    class Fixed(torch.nn.Module):
        def forward(self, x):
            return self.p

    net = Fixed()
    z = torch.ones(3, 6, 10, device="cuda")
    p = _x(3, 6, 10, 2, dtype=torch.float32)
    with fw.dual_level():
        net.p = fw.make_dual(p, torch.ones_like(p))
        u, v = guess.GuessModel(net).predict(z, z, z, z)
        ru, rv = guess.faces_from_cells(net.p)
        for a, r in ((u, ru), (v, rv)):
            assert torch.equal(a, r.double()) and torch.equal(fw.unpack_dual(a).tangent, fw.unpack_dual(r).tangent.double())
