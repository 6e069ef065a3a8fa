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
