"""ResNet-50's blocks and stages on the package's ops against the same model made of its modules."""

import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


class _Stage(nn.Sequential):
    """A stage that the model may not look into: its blocks are called, one output each."""


@pytest.mark.parametrize("form", ["pairs", "blocks"])
def test_blocks_match_their_modules(form, monkeypatch):
    """Gradients of the first stage pass every shortcut; fp32, where two orders of the same sums stay close."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fairring_b200.models import ResNet50

    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", False)
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", False)
    torch.manual_seed(0)
    model = ResNet50(num_classes=10, layers=(2, 2, 1, 1), width=8).cuda().to(memory_format=torch.channels_last)
    images = torch.randn(8, 3, 96, 96, device="cuda").contiguous(memory_format=torch.channels_last)
    labels = torch.randint(0, 10, (8,), device="cuda")
    start = {k: v.clone() for k, v in model.state_dict().items()}
    got = []
    for plain in (False, True):
        model.load_state_dict(start)
        if plain:  # a hook makes each module be called by itself
            for m in model.modules():
                m.register_forward_hook(lambda *a: None)
        elif form == "blocks":
            for name in ("layer1", "layer2", "layer3", "layer4"):
                setattr(model, name, _Stage(*getattr(model, name)))
        loss = model(images, labels)
        names = set()
        todo, seen = [loss.grad_fn], set()
        while todo:
            fn = todo.pop()
            if fn is not None and fn not in seen:
                seen.add(fn)
                names.add(type(fn).__name__)
                todo += [f for f, _ in fn.next_functions]
        assert ("_BatchNormActFnBackward" in names) != plain and ("_MaxPoolFnBackward" in names) != plain
        grads = torch.autograd.grad(loss, list(model.parameters()))
        got.append([loss.detach(), *grads, *(b.clone() for b in model.buffers())])
    for a, b in zip(*got):
        if a.dtype == torch.long:
            assert torch.equal(a, b)
        else:  # sums of up to 8 x 48 x 48 terms in another order, through 18 layers
            assert float((a - b).norm()) <= 1e-3 * float(b.norm()) + 1e-6
