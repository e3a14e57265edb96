"""BatchNorm + residual + ReLU in one op against the same in fp64."""

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _reference(x, res, bn, relu, dy):
    leaves = [t.detach().double().requires_grad_(True) for t in (x, bn.weight, bn.bias)]
    r = None if res is None else res.detach().double().requires_grad_(True)
    z = F.batch_norm(leaves[0], None, None, leaves[1], leaves[2], True, 0.0, bn.eps)
    z = z if r is None else z + r
    y = F.relu(z) if relu else z
    grads = torch.autograd.grad(y, leaves + ([] if r is None else [r]), dy.double())
    return y.detach(), z.detach(), grads


def _close(got, want, eps, scale=0.0):
    """Within `eps` of the value (the type's rounding) plus 1e-4 of `scale` (fp32 sums and their inputs)."""
    bad = (got.double() - want).abs() > eps * want.abs() + 1e-4 * scale + 1e-12
    assert not bad.any(), (int(bad.sum()), float((got.double() - want).abs().max()))


# rows: 2 (the fewest), fewer than a block holds, remainders of the unrolled loops, more than one pass of the grid
@pytest.mark.parametrize("shape", [(2, 8, 1, 1), (3, 8, 5, 7), (2, 16, 9, 9), (4, 64, 33, 31), (8, 256, 14, 13),
                                   (16, 2048, 7, 7), (1, 2048, 1, 3), (16, 64, 112, 112)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("residual,relu", [(False, False), (False, True), (True, False), (True, True)])
def test_matches_fp64(shape, dtype, residual, relu):
    _need_gpu()
    from fairring_b200.ops import batch_norm_act
    from fairring_b200.ops.batchnorm import _fusable

    gen = torch.Generator(device="cuda").manual_seed(sum(shape))
    rand = lambda: torch.randn(shape, device="cuda", generator=gen).to(  # noqa: E731
        dtype=dtype, memory_format=torch.channels_last)
    offset = 3.0 * torch.arange(shape[1], device="cuda").view(1, -1, 1, 1).remainder(7)  # means far from zero
    x = (rand().float() + offset).to(dtype=dtype, memory_format=torch.channels_last).requires_grad_(True)
    res = rand().requires_grad_(True) if residual else None
    dy = rand()
    bn = nn.BatchNorm2d(shape[1], device="cuda")
    with torch.no_grad():
        bn.weight.normal_(1.0, 0.2, generator=gen)
        bn.bias.normal_(0.0, 0.5, generator=gen)
    want_stats = nn.BatchNorm2d(shape[1], device="cuda").double()
    want_stats(x.detach().double())

    assert _fusable(bn, x, res)
    y = batch_norm_act(bn, x, res, nn.ReLU(inplace=True) if relu else None)
    y_ref, z, grads_ref = _reference(x, res, bn, relu, dy)
    grads = torch.autograd.grad(y, [x, bn.weight, bn.bias] + ([res] if residual else []), dy)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    _close(y, y_ref, eps, 1.0)
    # elements whose sign the rounding of z decides are left out, and where one is left out its channel's sums are off
    sure = (z.abs() > 1e-4) if relu else torch.ones_like(z, dtype=torch.bool)
    unsure = (~sure).sum((0, 2, 3)).double()
    n = x.numel() / shape[1]
    slack = 4.0 * float((unsure / n).max()) * float(dy.abs().max())
    wide = max(1.0, float(grads_ref[0].abs().max()))
    bad = ((grads[0].double() - grads_ref[0]).abs() > eps * grads_ref[0].abs() + 1e-4 * wide + slack * wide) & sure
    assert not bad.any(), int(bad.sum())
    for got, want in zip(grads[1:3], grads_ref[1:3]):
        assert ((got.double() - want).abs() <= 1e-4 * n ** 0.5 * 10 + 8.0 * unsure * float(dy.abs().max())).all()
    if residual:
        assert ((grads[3].double() - grads_ref[3]).abs()[sure] <= 1e-12).all()  # dy or zero: exact
    _close(bn.running_mean, want_stats.running_mean, 2.0 ** -22, 1e-2)
    _close(bn.running_var, want_stats.running_var, 2.0 ** -20, 1e-2)
    assert int(bn.num_batches_tracked) == 1


def test_a_channel_far_from_zero_keeps_its_variance():
    """Standard deviation 1 around a mean of 1000, with an outlier in front."""
    _need_gpu()
    from fairring_b200.ops import batch_norm_act

    x = torch.randn(32, 64, 28, 28, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) + 1000
    x[0, :, 0, 0] += 300
    x = x.contiguous(memory_format=torch.channels_last)
    bn = nn.BatchNorm2d(64, device="cuda", momentum=1.0)
    batch_norm_act(bn, x)
    want = x.double().var((0, 2, 3))
    assert ((bn.running_var.double() - want).abs() <= 1e-5 * want).all()


def test_nan_passes_the_relu():
    """As in torch: NaN stays NaN forward, and a gradient passes where the output is NaN."""
    _need_gpu()
    from fairring_b200 import _C

    x = torch.randn(2, 8, 4, 4, device="cuda").contiguous(memory_format=torch.channels_last)
    x[0, 3, 1, 1] = float("nan")  # its channel's statistics are NaN
    res = torch.randn_like(x)
    bn, relu = nn.BatchNorm2d(8, device="cuda"), nn.ReLU()
    from fairring_b200.ops import batch_norm_act

    y, want = batch_norm_act(bn, x, res, relu), relu(nn.BatchNorm2d(8, device="cuda")(x) + res)
    assert torch.equal(y.isnan(), want.isnan()) and bool(y[:, 3].isnan().all()) and int(y.isnan().sum()) == 32
    ones, stat = torch.ones_like(x), torch.ones(8, device="cuda")
    dz = _C.batch_norm_bwd(ones, torch.zeros_like(x), y.detach(), bn.weight.detach(), bn.bias.detach(), stat, stat, True)[1]
    assert torch.equal(dz, (~(y <= 0)).float())


def test_calls_the_modules_where_they_cannot_be_skipped():
    _need_gpu()
    from fairring_b200.ops import batch_norm_act
    from fairring_b200.ops.batchnorm import _fusable

    x = torch.randn(4, 16, 6, 6, device="cuda").contiguous(memory_format=torch.channels_last)
    bn, relu = nn.BatchNorm2d(16, device="cuda"), nn.ReLU()
    assert _fusable(bn, x, None)
    assert not _fusable(bn, x.contiguous(), None)  # NCHW
    assert not _fusable(bn, x.half(), None)
    assert not _fusable(bn, x, x.bfloat16())
    for channels in (24, 4096):  # no power of two, too many
        wide = torch.zeros(2, channels, 4, 4, device="cuda").contiguous(memory_format=torch.channels_last)
        assert not _fusable(nn.BatchNorm2d(channels, device="cuda"), wide, None)
    seen = []
    handle = relu.register_forward_hook(lambda *a: seen.append(1))
    batch_norm_act(bn, x, relu=relu)
    assert seen == [1]
    handle.remove()
    bn.eval()
    torch.testing.assert_close(batch_norm_act(bn, x, relu=relu), relu(bn(x)))


def test_second_derivative():
    _need_gpu()
    from fairring_b200.ops import batch_norm_act

    torch.manual_seed(0)
    x0 = torch.randn(3, 8, 4, 4, device="cuda").contiguous(memory_format=torch.channels_last)
    got = []
    for fused in (True, False):
        x = x0.clone(memory_format=torch.channels_last).requires_grad_(True)
        bn = nn.BatchNorm2d(8, device="cuda")
        y = batch_norm_act(bn, x) if fused else bn(x)
        (g,) = torch.autograd.grad((y ** 3).sum(), x, create_graph=True)
        got.append(torch.autograd.grad((g ** 2).sum(), x)[0])
    torch.testing.assert_close(got[0], got[1], rtol=1e-3, atol=1e-4 * float(got[1].abs().max()))


@pytest.mark.parametrize("residual", ["none", "other", "same"])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("twice", [True, False])
def test_second_derivative_with_all_that_follows(residual, relu, twice):
    """`same`: the input itself as the residual, whose gradient must not be counted twice."""
    _need_gpu()
    from fairring_b200.ops import batch_norm_act

    torch.manual_seed(1)
    x0, r0 = (torch.randn(3, 8, 4, 4, device="cuda").contiguous(memory_format=torch.channels_last) for _ in range(2))
    act, got = nn.ReLU() if relu else None, []
    for fused in (True, False):
        x, r = (t.clone(memory_format=torch.channels_last).requires_grad_(True) for t in (x0, r0))
        bn = nn.BatchNorm2d(8, device="cuda")
        a = x * 1.0
        res = {"none": None, "other": r * 1.0, "same": a}[residual]
        if fused:
            y, y2 = batch_norm_act(bn, a, res, act, twice=True) if twice else (batch_norm_act(bn, a, res, act),) * 2
        else:
            z = bn(a) if res is None else bn(a) + res
            y = y2 = act(z) if relu else z
        leaves = [x, bn.weight, bn.bias] + ([r] if residual == "other" else [])
        first = torch.autograd.grad((y ** 3).sum() + (y2 ** 2).sum(), leaves, create_graph=True)
        got.append([*first, *torch.autograd.grad(sum((g ** 2).sum() for g in first), leaves)])
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-4 * float(b.detach().abs().max()))


@pytest.mark.parametrize("pin", [False, True])
def test_saved_tensors_that_come_back_in_another_layout(pin):
    _need_gpu()
    from fairring_b200.ops import batch_norm_act

    x0, r0, dy = (torch.randn(3, 16, 5, 7, device="cuda").contiguous(memory_format=torch.channels_last) for _ in range(3))
    bn, got = nn.BatchNorm2d(16, device="cuda"), []
    for hooks in (torch.autograd.graph.save_on_cpu(pin_memory=pin), torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t)):
        x, r = x0.clone(memory_format=torch.channels_last).requires_grad_(True), r0.clone(memory_format=torch.channels_last).requires_grad_(True)
        with hooks:
            y = batch_norm_act(bn, x, r, nn.ReLU())
        got.append(torch.autograd.grad(y, [x, r, bn.weight, bn.bias], dy))
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_the_residual_is_not_kept():
    _need_gpu()
    import weakref

    from fairring_b200.ops import batch_norm_act

    x = torch.randn(4, 16, 6, 6, device="cuda").contiguous(memory_format=torch.channels_last).requires_grad_(True)
    res = x.detach().clone(memory_format=torch.channels_last)
    y = batch_norm_act(nn.BatchNorm2d(16, device="cuda"), x, res, nn.ReLU())
    gone = weakref.ref(res)
    del res
    assert gone() is None and y.requires_grad


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("residual,relu", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("use", ["both", "first", "second"])
def test_two_uses_of_the_output(dtype, residual, relu, use):
    _need_gpu()
    from fairring_b200.ops import batch_norm_act

    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda: torch.randn(4, 64, 13, 11, device="cuda", generator=gen).to(  # noqa: E731
        dtype=dtype, memory_format=torch.channels_last)
    x, res, dy, dy2 = rand().requires_grad_(True), rand().requires_grad_(True) if residual else None, rand(), rand()
    bn, act = nn.BatchNorm2d(64, device="cuda"), nn.ReLU() if relu else None
    inputs = [x, bn.weight, bn.bias] + ([res] if residual else [])
    pair = batch_norm_act(bn, x, res, act, twice=True)
    outs = {"both": (list(pair), [dy, dy2]), "first": ([pair[0]], [dy]), "second": ([pair[1]], [dy2])}[use]
    got = torch.autograd.grad(outs[0], inputs, outs[1])
    y = batch_norm_act(bn, x, res, act)
    assert torch.equal(pair[0], y) and torch.equal(pair[1], y)
    total = sum(d.double() for d in outs[1])
    want = _reference(x, res, bn, relu, total)[2]
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
    far = 2.0 ** -7 if dtype == torch.bfloat16 else 1e-5  # the sum of two gradients is rounded before it is used
    for g, w in zip(got, want):
        assert float((g.double() - w).norm()) <= (eps + far) * float(w.norm())
