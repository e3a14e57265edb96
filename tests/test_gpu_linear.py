"""GELU and bias gradients around bf16 linear layers, against fp64."""

import sys

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# one thread across, a ragged block, one full block of 2048 columns and a second one; one row, remainders
# of the unrolled loop, one and many strips
@pytest.mark.parametrize("cols", [8, 120, 512, 2048, 2056, 8192])
@pytest.mark.parametrize("rows", [1, 7, 333, 4099])
@pytest.mark.parametrize("form", ["none", "tanh"])
def test_gelu_and_column_sums(rows, cols, form):
    _need_gpu()
    from fairring_b200 import _C

    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda", generator=gen) * 3).bfloat16()
    dy = torch.randn(rows, cols, device="cuda", generator=gen).bfloat16()
    ref = x.double().requires_grad_(True)
    want = F.gelu(ref, approximate=form)
    (want_dx,) = torch.autograd.grad(want, ref, dy.double())
    y = _C.gelu_fwd(x, form == "tanh")
    dx, db = _C.gelu_bwd(dy, x, form == "tanh", torch.float32)
    for got, w in ((y, want), (dx, want_dx)):  # bf16, and fp32's cancellation in 1 + erf for negative x
        assert ((got.double() - w).abs() <= 2.0 ** -8 * w.abs() + 2e-6).all()
    assert ((db.double() - want_dx.sum(0)).abs() <= 1e-5 * rows ** 0.5 + 2e-6).all()
    plain = _C.column_sum(dy, torch.float32)
    assert ((plain.double() - dy.double().sum(0)).abs() <= 1e-5 * rows ** 0.5).all()
    low = _C.column_sum(dy, torch.bfloat16)
    assert torch.equal(low, plain.bfloat16())


@pytest.mark.parametrize("form", ["none", "tanh"])
def test_gelu_of_the_largest_values(form):
    """Infinities, NaN and the largest finite values give what torch gives, NaN included."""
    _need_gpu()
    from fairring_b200 import _C

    big = torch.finfo(torch.bfloat16).max
    x = torch.tensor([float("inf"), float("-inf"), float("nan"), big, -big, 1e4, -1e4, 0.0], device="cuda").bfloat16().view(1, 8)
    ref = x.detach().requires_grad_(True)
    want = F.gelu(ref, approximate=form)
    (want_dx,) = torch.autograd.grad(want, ref, torch.ones_like(x))
    torch.testing.assert_close(_C.gelu_fwd(x, form == "tanh"), want, rtol=0, atol=0, equal_nan=True)
    got = _C.gelu_bwd(torch.ones_like(x), x, form == "tanh", torch.float32)[0]
    torch.testing.assert_close(got, want_dx, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("weights", [torch.float32, torch.bfloat16])
def test_layers_match_torch(weights, monkeypatch):
    _need_gpu()
    from fairring_b200.ops import linear, linear_gelu

    monkeypatch.setattr(sys.modules[linear.__module__], "_FUSE_FROM", 1)

    torch.manual_seed(0)
    fc = nn.Linear(64, 136, device="cuda", dtype=weights)
    x = torch.randn(3, 50, 64, device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn(3, 50, 136, device="cuda").bfloat16()
    for ours, theirs in ((linear, lambda m, t: m(t)), (linear_gelu, lambda m, t: F.gelu(m(t)))):
        got = []
        for f in (ours, theirs):
            with torch.autocast("cuda", dtype=torch.bfloat16, enabled=weights == torch.float32):
                y = f(fc, x)
            assert y.dtype == torch.bfloat16
            got.append([y, *torch.autograd.grad(y, [x, fc.weight, fc.bias], dy)])
        for a, b in zip(*got):
            assert a.dtype == b.dtype and a.shape == b.shape
            scale = float(b.detach().float().abs().max())
            torch.testing.assert_close(a.float(), b.float(), rtol=2.0 ** -6, atol=2.0 ** -7 * scale)


def test_the_layer_is_called_where_it_cannot_be_skipped(monkeypatch):
    _need_gpu()
    from fairring_b200.ops import linear

    module = sys.modules[linear.__module__]
    _fusable = module._fusable
    with torch.autocast("cuda", dtype=torch.bfloat16):
        edge = nn.Linear(8, 1024, device="cuda")
        assert _fusable(edge, torch.zeros(4096, 8, device="cuda"))
        assert not _fusable(edge, torch.zeros(4095, 8, device="cuda"))
    monkeypatch.setattr(module, "_FUSE_FROM", 1)
    fc = nn.Linear(16, 24, device="cuda")
    x = torch.randn(4, 16, device="cuda")
    assert not _fusable(fc, x)  # fp32 without autocast
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert _fusable(fc, x)
        seen = []
        handle = fc.register_forward_hook(lambda *a: seen.append(1))
        linear(fc, x)
        assert seen == [1]
        handle.remove()
        (g,) = torch.autograd.grad(linear(fc, x.requires_grad_(True)).float().pow(2).sum(), fc.bias, create_graph=True)
        assert g.requires_grad
