"""Which tensors the one-pass kernels of the learned guess are given (host
checks; a stand-in library records the calls)."""
import pytest
import torch

from glide_b200 import _native as N
from glide_b200 import guess


class Recorder:
    """Accepts every shape; remembers the entry points called and their arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*a):
            self.calls.append((name, a))
            return 1 if name == "glide_conv3x3_rows_ok" else 0
        return call

    def args(self, name):
        return [a for n, a in self.calls if n == name]


@pytest.fixture
def lib(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(guess, "_lib", lambda: r)
    monkeypatch.setattr(N, "stream_handle", lambda stream=None: None)
    return r


def _layer(Cin=32, Cout=32, dtype=torch.bfloat16, width=None):
    return (torch.zeros(1, 4, 64, Cin, dtype=dtype), torch.zeros(Cout, width or 9 * Cin), torch.zeros(Cout))


def test_conv_takes_the_row_march(lib):
    guess.conv3x3_relu(*_layer())
    assert len(lib.args("glide_conv3x3_rows_f32w")) == 1


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_conv_refuses_other_activation_types(lib, dtype):
    with pytest.raises(AssertionError):
        guess.conv3x3_relu(*_layer(dtype=dtype))
    assert not lib.args("glide_conv3x3_rows_f32w")


@pytest.mark.parametrize("width", [9 * 32 - 8, 9 * 16, 9 * 32 + 16])
def test_conv_passes_the_width_of_the_weights_on(lib, width):
    """Weights narrower or wider than 9 Cin reach the entry point that takes
    their pitch: it refuses the narrow ones and reads the padded ones right."""
    guess.conv3x3_relu(*_layer(width=width))
    assert not lib.args("glide_conv3x3_rows_f32w")
    (a,) = lib.args("glide_conv3x3_bf16")
    assert a[6] == width


@pytest.mark.parametrize("b", [torch.zeros(32, dtype=torch.float64), torch.zeros(64)[::2], torch.zeros(31)])
def test_conv_row_march_needs_a_plain_bias(lib, b):
    x, W, _ = _layer()
    guess.conv3x3_relu(x, W, b)
    assert not lib.args("glide_conv3x3_rows_f32w")


def _sources(h=2, w=32, C0=32, C1=32, dtype=torch.bfloat16, **skip):
    s = dict(Bn=1, H=2 * h, W=2 * w, C=C1, dtype=dtype) | skip
    return (torch.zeros(1, h, w, C0, dtype=dtype), torch.zeros(s["Bn"], s["H"], s["W"], s["C"], dtype=s["dtype"]),
            torch.zeros(32, 9 * (C0 + s["C"])), torch.zeros(32))


def test_two_sources_are_read_in_place(lib):
    guess.conv3x3_up_cat(*_sources())
    (a,) = lib.args("glide_conv3x3_rows_f32w")
    assert a[2] == 1 and a[4] == 32


@pytest.mark.parametrize("skip", [dict(Bn=2), dict(H=6), dict(W=66), dict(W=128), dict(H=3)])
def test_two_sources_of_unequal_sizes_are_refused(lib, skip):
    """As torch.cat refuses them."""
    with pytest.raises(RuntimeError):
        guess.conv3x3_up_cat(*_sources(**skip))
    assert not [n for n, _ in lib.calls if n.startswith("glide_conv3x3") and n != "glide_conv3x3_rows_ok"]


@pytest.mark.parametrize("x,skip", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                    (torch.float16, torch.bfloat16)])
def test_two_sources_of_other_types_are_refused(lib, x, skip):
    a, s, W, b = _sources(dtype=x)
    with pytest.raises(AssertionError):
        guess.conv3x3_up_cat(a, s.to(skip), W, b)
    assert not lib.args("glide_conv3x3_rows_f32w") and not lib.args("glide_conv3x3_cat_bf16")


@pytest.mark.parametrize("which", ["x", "skip", "no skip channels", "padded weights"])
def test_two_sources_that_need_the_joined_tensor(lib, which):
    """What only the concatenation can serve still runs on it."""
    x, skip, W, b = _sources(C1=0) if which == "no skip channels" else _sources()

    def shifted(t):   # contiguous, 2 bytes off a 16-byte boundary
        return torch.zeros(t.numel() + 1, dtype=t.dtype)[1:].view(t.shape)

    if which == "x":
        x = shifted(x)
    if which == "skip":
        skip = shifted(skip)
    if which == "padded weights":
        W = torch.zeros(32, W.shape[1] + 8)
    guess.conv3x3_up_cat(x, skip, W, b)
    assert not lib.args("glide_conv3x3_cat_bf16") and all(a[3] is None for a in lib.args("glide_conv3x3_rows_f32w"))
    assert lib.args("glide_conv3x3_rows_f32w") or lib.args("glide_conv3x3_bf16")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
def test_pool_on_the_host_is_torch(lib, dtype):
    x = torch.arange(1 * 4 * 6 * 8, dtype=torch.float32).view(1, 4, 6, 8).to(dtype)
    ref = torch.nn.functional.avg_pool2d(x.float().permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1)
    assert torch.equal(guess._pool(x), ref.to(torch.bfloat16)) and not lib.calls


@pytest.mark.parametrize("shape", [(1, 3, 4, 8), (1, 4, 5, 8)])
def test_pool_refuses_odd_sizes(lib, shape):
    with pytest.raises(RuntimeError):
        guess._pool(torch.zeros(shape, dtype=torch.bfloat16))
    assert not lib.calls


def test_pool_of_an_empty_batch(lib):
    assert guess._pool(torch.zeros(0, 4, 4, 8, dtype=torch.bfloat16)).shape == (0, 2, 2, 8) and not lib.calls
