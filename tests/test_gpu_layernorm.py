"""The LayerNorm kernels at the edges of their warps and rounds, against fp64."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# A block of 256 threads does a row, 8 columns to a thread, in up to four rounds of 2048: one thread, a warp
# less one thread, a full warp and one thread more, several warps, a full round and one thread of the next, four
# rounds less one thread and all four; one row, fewer rows than blocks, more rows than blocks
@pytest.mark.parametrize("cols", [8, 248, 256, 264, 768, 1032, 2048, 2056, 8184, 8192])
@pytest.mark.parametrize("rows", [1, 5, 3001])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_layer_norm_against_fp64(cols, rows, dtype):
    _need_gpu()
    from fairring_b200.ops import fused_layer_norm

    gen = torch.Generator(device="cuda").manual_seed(cols + rows)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x = (rand(rows, cols) * 2 + 0.5).to(dtype).requires_grad_(True)
    w, b = rand(cols).requires_grad_(True), rand(cols).requires_grad_(True)
    dy = rand(rows, cols).to(dtype)
    y = fused_layer_norm(x, w, b)
    grads = torch.autograd.grad(y, [x, w, b], dy)
    leaves = [t.detach().double().requires_grad_(True) for t in (x, w, b)]
    want = F.layer_norm(leaves[0], (cols,), leaves[1], leaves[2], 1e-5)
    wants = torch.autograd.grad(want, leaves, dy.double())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
    for got, ref in zip([y, grads[0]], [want, wants[0]]):  # a rounding of the type, and of the fp32 terms of the sum
        assert ((got.double() - ref).abs() <= eps * ref.abs() + 4e-6 * max(1.0, float(ref.abs().max()))).all()
    for got, ref in zip(grads[1:], wants[1:]):  # fp32 sums over the rows
        assert ((got.double() - ref).abs() <= 1e-5 * (rows ** 0.5 + 1) * 4).all()


def test_rows_off_a_16_byte_boundary():
    _need_gpu()
    from fairring_b200.ops import fused_layer_norm

    x = torch.randn(5 * 64 + 1, device="cuda")[1:].view(5, 64)
    w, b = torch.ones(65, device="cuda")[1:], torch.zeros(65, device="cuda")[1:]
    torch.testing.assert_close(fused_layer_norm(x, w, b), F.layer_norm(x, (64,)), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("kind", ["norm", "transposed", "bf16", "residual", "residual bf16"])
def test_second_derivative(kind, native, monkeypatch):
    _need_gpu()
    import sys

    from fairring_b200.ops import FusedLayerNorm, add_layer_norm

    if not native:
        monkeypatch.setattr(sys.modules[FusedLayerNorm.__module__], "plain_autograd", lambda: False)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x0, br0 = torch.randn(24, 24, device="cuda", generator=gen), torch.randn(24, 24, device="cuda", generator=gen)
    low = kind.endswith("bf16")
    if low:
        br0 = br0.bfloat16()
        x0 = x0.bfloat16() if kind == "bf16" else x0
    got = []
    for fused in (True, False):
        norm = (FusedLayerNorm if fused else torch.nn.LayerNorm)(24, device="cuda")
        x, br = x0.clone().requires_grad_(True), br0.clone().requires_grad_(True)
        if kind.startswith("residual"):
            stream = x + br
            stream, y = add_layer_norm(norm, x, br) if fused else (stream, norm(stream))
            out, leaves = (y ** 3).sum() + (stream ** 3).sum(), [x, br, norm.weight, norm.bias]
        else:
            a = x.t() if kind == "transposed" else x
            y = norm(a) if fused else F.layer_norm(a.float(), (24,), norm.weight, norm.bias).to(a.dtype)
            out, leaves = (y.float() ** 3).sum(), [x, norm.weight, norm.bias]
        first = torch.autograd.grad(out, leaves, create_graph=True)
        assert all(g.requires_grad for g in first)
        got.append([*first, *torch.autograd.grad(sum((g.float() ** 2).sum() for g in first), leaves)])
    rtol = 2.0 ** -5 if low else 1e-3  # up to four roundings of the type on the way
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=rtol, atol=rtol * float(b.detach().abs().max()))


@pytest.mark.parametrize("kind", ["norm", "residual", "pair"])
def test_no_rows(kind):
    """An empty batch gives parameter gradients of zero."""
    _need_gpu()
    from fairring_b200.ops import FusedLayerNorm, add_layer_norm

    norm = FusedLayerNorm(2048, device="cuda")
    x, br = (torch.empty(0, 2048, device="cuda", requires_grad=True) for _ in range(2))
    junk = [torch.full((2048,), 7.0, device="cuda") for _ in range(8)]  # what the allocator hands out next
    del junk
    if kind == "pair":
        from fairring_b200 import _C

        d = torch.empty(0, 2048, device="cuda")
        stat = torch.empty(0, device="cuda")
        _, _, dw, db = _C.add_layer_norm_bwd(None, d, norm.weight.detach(), stat, stat, None, False, d)
    else:
        y = norm(x) if kind == "norm" else add_layer_norm(norm, x, br)[1]
        dx, dw, db = torch.autograd.grad(y.sum(), [x, norm.weight, norm.bias])
        assert dx.shape == x.shape
    assert not dw.any() and not db.any()


# a warp's columns and part of another's, all warps', ragged second and third rounds
@pytest.mark.parametrize("cols", [8, 264, 2048, 4104, 8192])
@pytest.mark.parametrize("kind", ["norm", "residual"])
@pytest.mark.parametrize("row", ["far", "outlier", "far and outlier", "constant"])
def test_a_mean_far_from_zero_keeps_the_variance(cols, kind, row):
    _need_gpu()
    from fairring_b200.ops import FusedLayerNorm, add_layer_norm

    gen = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(64, cols, device="cuda", generator=gen)
    if row == "constant":
        x[:] = 1000.0
    if row.startswith("far"):
        x += 1000
    if row.endswith("outlier"):
        x[:, 0] += 500.0  # the element that the differences are taken from
    norm = FusedLayerNorm(cols, device="cuda")
    y = norm(x) if kind == "norm" else add_layer_norm(norm, x, torch.zeros_like(x))[1]
    # the mean is known to a few of fp32's steps at 1000 (6e-5), everything else to a few of its own
    assert float((y.double() - F.layer_norm(x.double(), (cols,))).abs().max()) < 2e-4


def test_a_row_that_is_not_finite():
    _need_gpu()
    from fairring_b200.ops import FusedLayerNorm

    norm = FusedLayerNorm(512, device="cuda")
    x = torch.randn(6, 512, device="cuda")
    x[0, 0], x[1, 300], x[2, 511], x[3, 0] = float("inf"), float("-inf"), float("nan"), float("nan")
    assert torch.equal(norm(x).isnan().all(1), torch.tensor([1, 1, 1, 1, 0, 0], device="cuda", dtype=torch.bool))
