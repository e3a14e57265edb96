"""The cross-entropy kernels at the edges of their rows' parts, against fp64."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _check(logits, leaf, loss, targets):
    """Against fp64 on the same logits: 20 roundings of the sums, one of the result's type, and what a
    relative error of 2**-21 in exp() (its fast form over the range that matters) makes of a probability."""
    ref = leaf.detach().double().requires_grad_(True)
    want = F.cross_entropy(ref, targets.where(targets >= 0, -100))
    assert abs(float(loss.detach()) - float(want.detach())) <= 3e-6 * max(1.0, float(ref.detach()[ref.isfinite()].abs().max()))
    (loss * 1.7).backward()
    want_grad = torch.autograd.grad(want * 1.7, ref)[0]
    n = max(1, int((targets >= 0).sum()))
    eps = 2.0 ** -8 if leaf.dtype == torch.bfloat16 else 2.0 ** -20
    bad = (leaf.grad.double() - want_grad).abs() > eps * want_grad.abs() + 3e-6 * 1.7 / n
    assert not bad.any(), int(bad.sum())


# one thread's worth, remainders on both sides of the 16-byte vectors, the batch of the narrow block
# (128 x 4 vectors) and of the wide one (256 x 4), where the wide block takes over, two pieces of the backward
@pytest.mark.parametrize("vocab", [1, 7, 8, 9, 1000, 1001, 4095, 4097, 8191, 8192, 8193, 16383, 16384, 16385, 50265])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_every_row_length(vocab, dtype):
    _need_gpu()
    from fairring_b200.ops import fused_cross_entropy

    gen = torch.Generator(device="cuda").manual_seed(vocab)
    rows = 19  # odd rows of an odd vocabulary start at every offset from a 16-byte boundary
    leaf = (torch.randn(rows, vocab, device="cuda", generator=gen) * 3).to(dtype).requires_grad_(True)
    targets = torch.randint(0, vocab, (rows,), device="cuda", generator=gen)
    targets[3], targets[4], targets[5] = -100, 0, vocab - 1
    logits = leaf * 1.0
    before = logits.detach().clone()
    loss = fused_cross_entropy(logits, targets)
    _check(logits, leaf, loss, targets)
    assert float(leaf.grad[3].abs().sum()) == 0.0
    if vocab % 8:  # only a vocabulary that is a multiple of 8 consumes its logits
        assert torch.equal(logits, before)


@pytest.mark.parametrize("vocab", [1000, 1001, 20000])
@pytest.mark.parametrize("fill", [float("-inf"), "lowest"])
def test_masked_logits(vocab, fill):
    _need_gpu()
    from fairring_b200.ops import fused_cross_entropy

    for dtype in (torch.bfloat16, torch.float32):
        value = torch.finfo(dtype).min if fill == "lowest" else fill
        base = torch.randn(6, vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(vocab))
        base = base.to(dtype)
        base[:, 1:] = torch.where(torch.rand(6, vocab - 1, device="cuda") < 0.5, base[:, 1:], value)
        base[2, 1:] = value  # a single logit left
        base[3, : vocab // 2 + 1] = value  # whole threads without one
        base[3, -1] = 1.0
        targets = torch.zeros(6, dtype=torch.long, device="cuda")
        targets[3] = vocab - 1
        leaf = base.clone().requires_grad_(True)
        loss = fused_cross_entropy(leaf * 1.0, targets)
        ref = base.double().requires_grad_(True)
        want = F.cross_entropy(ref, targets)
        assert abs(float(loss) - float(want)) < 1e-5
        loss.backward()
        assert bool(leaf.grad.isfinite().all())
        torch.testing.assert_close(leaf.grad.double(), torch.autograd.grad(want, ref)[0], rtol=2.0 ** -8, atol=1e-6)


def test_rows_off_a_16_byte_boundary():
    _need_gpu()
    from fairring_b200.ops import fused_cross_entropy

    store = torch.randn(5 * 1024 + 3, device="cuda")
    leaf = store.clone().requires_grad_(True)
    logits = (leaf * 1.0)[3:].view(5, 1024)
    targets = torch.tensor([0, 1, 1022, 1023, -1], device="cuda")
    loss = fused_cross_entropy(logits, targets)
    ref = store[3:].view(5, 1024).double()
    assert abs(float(loss) - float(F.cross_entropy(ref[:4], targets[:4]))) < 1e-5
    loss.backward()
    r = ref.clone().requires_grad_(True)
    F.cross_entropy(r[:4], targets[:4]).backward()
    torch.testing.assert_close(leaf.grad[3:].view(5, 1024).double(), r.grad, rtol=1e-5, atol=1e-7)


def test_no_counted_row_and_second_derivative():
    _need_gpu()
    from fairring_b200.ops import fused_cross_entropy

    ignored = torch.full((4,), -100, device="cuda")
    assert float(fused_cross_entropy(torch.randn(4, 16, device="cuda"), ignored)) == 0.0
    assert torch.isnan(fused_cross_entropy(torch.randn(4, 17, device="cuda"), ignored))  # as torch's own loss
    x = torch.randn(4, 17, device="cuda", requires_grad=True)
    t = torch.tensor([1, 2, -100, 16], device="cuda")
    got = []
    for f in (fused_cross_entropy, F.cross_entropy):
        (g,) = torch.autograd.grad(f(x, t), x, create_graph=True)
        got.append(torch.autograd.grad((g ** 2).sum(), x)[0])
    torch.testing.assert_close(got[0], got[1], rtol=1e-4, atol=1e-6)


# the vocabulary of the gradient over the logits, and one that keeps them
@pytest.mark.parametrize("vocab", [16, 17])
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_second_derivative_and_the_logits_behind_it(vocab, native, dtype, monkeypatch):
    _need_gpu()
    import sys

    from fairring_b200.ops import fused_cross_entropy

    if not native:
        monkeypatch.setattr(sys.modules[fused_cross_entropy.__module__], "plain_autograd", lambda: False)
    leaf = torch.randn(5, vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(vocab)).to(dtype)
    t = torch.tensor([1, -100, 0, vocab - 1, 2], device="cuda")
    got = []
    for f in (fused_cross_entropy, lambda a, b: F.cross_entropy(a.float(), b)):
        x = leaf.clone().requires_grad_(True)
        logits = x * 1.0
        before = logits.detach().clone()
        loss = f(logits, t)
        (g,) = torch.autograd.grad(loss * loss, x, create_graph=True)
        assert g.requires_grad and torch.equal(logits, before)
        got.append([g, torch.autograd.grad((g.float() ** 2).sum(), x)[0]])
    rtol = 2.0 ** -6 if dtype == torch.bfloat16 else 1e-4  # two to three roundings on the way
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=rtol, atol=rtol * float(b.detach().abs().max()))


@pytest.mark.parametrize("vocab", [1000, 1001, 50257])
def test_fp32_gradients_are_as_exact_as_torch(vocab):
    """Logits as a trained head has them, far apart: exp() of differences down to -40."""
    _need_gpu()
    from fairring_b200.ops import fused_cross_entropy

    gen = torch.Generator(device="cuda").manual_seed(vocab)
    x = torch.randn(512, vocab, device="cuda", generator=gen) * 5
    t = torch.randint(0, vocab, (512,), device="cuda", generator=gen)
    ref = x.double().requires_grad_(True)
    want = F.cross_entropy(ref, t)
    (wg,) = torch.autograd.grad(want, ref)
    wg.scatter_(1, t[:, None], 0.0)  # the probabilities alone: the target's entry is 1 minus one
    error = []
    for f in (fused_cross_entropy, F.cross_entropy):
        leaf = x.clone().requires_grad_(True)
        (g,) = torch.autograd.grad(f(leaf * 1.0, t), leaf)
        error.append(float((g.double().scatter_(1, t[:, None], 0.0) - wg).norm() / wg.norm()))
    # both round the argument of exp() and its result; torch's own sum and logarithm may fall on either side
    assert error[0] <= 1.2 * error[1] + 2.0 ** -24, error


def test_padding_behind_the_classes():
    """Targets at the edges of what is allowed; one outside would fail an assertion on the GPU."""
    _need_gpu()
    from fairring_b200 import _C
    from fairring_b200.ops import cross_entropy_keeping_logits

    base = torch.randn(4, 24, device="cuda")
    base[:, 19:] = float("-inf")
    targets = torch.tensor([0, 18, -100, 7], device="cuda")
    x = base.clone().requires_grad_(True)
    loss = cross_entropy_keeping_logits(x, targets, 19)
    ref = base[:, :19].double().requires_grad_(True)
    want = F.cross_entropy(ref, targets)
    assert abs(float(loss) - float(want)) < 1e-5
    (g,) = torch.autograd.grad(loss, x)
    assert not g[:, 19:].any()
    torch.testing.assert_close(g[:, :19].double(), torch.autograd.grad(want, ref)[0], rtol=1e-5, atol=1e-6)
    with pytest.raises(RuntimeError):
        _C.cross_entropy(base, targets, 25)
