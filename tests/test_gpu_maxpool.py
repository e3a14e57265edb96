"""Max pooling against torch: the same elements chosen, ties and NaN included."""

import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# windows that touch, overlap and leave gaps, with and without padding; inputs that they divide into and not
@pytest.mark.parametrize("window,stride,pad", [(3, 2, 1), (2, 2, 0), (3, 1, 1), (2, 3, 1), (5, 2, 2), (1, 1, 0), (16, 4, 8)])
@pytest.mark.parametrize("shape", [(1, 8, 16, 16), (3, 24, 17, 23), (2, 64, 112, 56)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_matches_torch(shape, window, stride, pad, dtype):
    _need_gpu()
    from fairring_b200.ops import max_pool

    gen = torch.Generator(device="cuda").manual_seed(window + shape[1])
    x = torch.randint(-3, 4, shape, device="cuda", generator=gen).to(dtype)  # few values: many ties
    x = x.contiguous(memory_format=torch.channels_last).requires_grad_(True)
    pool = nn.MaxPool2d(window, stride, pad)
    y, want = max_pool(pool, x), pool(x)
    assert type(y.grad_fn).__name__ == "_MaxPoolFnBackward"
    assert torch.equal(y, want) and y.is_contiguous(memory_format=torch.channels_last)
    # whole numbers whose sums are exact in either type
    dy = torch.randint(-2, 3, want.shape, device="cuda", generator=gen).to(dtype)
    got, ref = torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(want, x, dy)[0]
    assert torch.equal(got, ref)


def test_nan_and_infinities():
    _need_gpu()
    from fairring_b200.ops import max_pool

    x = torch.randn(2, 8, 12, 12, device="cuda").contiguous(memory_format=torch.channels_last)
    x[0, :, 3, 3], x[0, :, 4, 4], x[1, :, :, :] = float("nan"), float("nan"), float("-inf")
    x.requires_grad_(True)
    pool = nn.MaxPool2d(3, 2, 1)
    # torch's NCHW form: in a window of -inf alone its channels-last form names element 0 of the image,
    # which need not lie in the window
    y, want = max_pool(pool, x), pool(x.contiguous())
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.nan_to_num(7.0), want.nan_to_num(7.0))
    dy = torch.ones_like(want)
    assert torch.equal(torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(want, x, dy)[0])


@pytest.mark.parametrize("pin", [False, True])
def test_saved_tensors_that_come_back_in_another_layout(pin):
    _need_gpu()
    from fairring_b200.ops import max_pool

    x = torch.randn(2, 8, 13, 12, device="cuda").contiguous(memory_format=torch.channels_last).requires_grad_(True)
    pool = nn.MaxPool2d(3, 2, 1)
    with torch.autograd.graph.save_on_cpu(pin_memory=pin):
        y = max_pool(pool, x)
    assert type(y.grad_fn).__name__ == "_MaxPoolFnBackward"
    dy = torch.randint(-2, 3, y.shape, device="cuda").float()
    assert torch.equal(torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(pool(x), x, dy)[0])


def test_calls_the_module_where_it_cannot_be_skipped():
    _need_gpu()
    from fairring_b200.ops import max_pool

    x = torch.randn(2, 8, 12, 12, device="cuda").contiguous(memory_format=torch.channels_last).requires_grad_(True)
    for pool in (nn.MaxPool2d(3, ceil_mode=True), nn.MaxPool2d((3, 2)), nn.MaxPool2d(3, dilation=2)):
        torch.testing.assert_close(max_pool(pool, x), pool(x))
    assert type(max_pool(nn.MaxPool2d(2), x.contiguous()).grad_fn).__name__ != "_MaxPoolFnBackward"  # NCHW
