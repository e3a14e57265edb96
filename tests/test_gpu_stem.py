"""The folded first convolution against torch's."""

import sys

import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# even and odd sizes, a single pixel, sizes smaller than the kernel
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (2, 5, 6), (3, 32, 32), (2, 33, 47), (1, 224, 223)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_matches_torch(n, h, w, dtype, monkeypatch):
    _need_gpu()
    from fairring_b200.ops import stem_conv

    monkeypatch.setattr(sys.modules[stem_conv.__module__], "_FOLD_FROM", 0)
    gen = torch.Generator(device="cuda").manual_seed(h)
    images = torch.randn(n, 3, h, w, device="cuda", generator=gen).to(dtype=dtype, memory_format=torch.channels_last)
    conv = nn.Conv2d(3, 16, 7, stride=2, padding=3, bias=False, device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y, want = stem_conv(conv, images), conv(images)
    assert type(y.grad_fn).__name__ == "_StemConvFnBackward"
    assert y.shape == want.shape and y.dtype == want.dtype
    # bf16 of fp32 sums of 147 products in another order
    ref = torch.nn.functional.conv2d(images.bfloat16().double(), conv.weight.detach().bfloat16().double(), None, 2, 3)
    assert float((y.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()) + 1e-5
    dy = torch.randn(want.shape, device="cuda", generator=gen).bfloat16().contiguous(memory_format=torch.channels_last)
    got, ref = torch.autograd.grad(y, conv.weight, dy)[0], torch.autograd.grad(want, conv.weight, dy)[0]
    assert got.dtype == ref.dtype and float((got - ref).norm()) <= 2.0 ** -7 * float(ref.norm())


def test_calls_the_module_where_it_cannot_be_skipped(monkeypatch):
    _need_gpu()
    from fairring_b200.ops import stem_conv

    images = torch.randn(2, 3, 16, 16, device="cuda").contiguous(memory_format=torch.channels_last)
    conv = nn.Conv2d(3, 16, 7, stride=2, padding=3, bias=False, device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert type(stem_conv(conv, images).grad_fn).__name__ != "_StemConvFnBackward"  # small
        monkeypatch.setattr(sys.modules[stem_conv.__module__], "_FOLD_FROM", 0)
        assert type(stem_conv(conv, images.contiguous()).grad_fn).__name__ != "_StemConvFnBackward"  # NCHW
        assert stem_conv(conv, images.clone().requires_grad_(True)).grad_fn.next_functions[0][0] is not None
    assert stem_conv(conv, images).dtype == torch.float32  # no autocast
