"""What looks through a model sees its modules: scripting, tracing, compilation, fake tensors, transforms."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.func import functional_call, grad, jvp
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils.flop_counter import FlopCounterMode

from fairring_b200.models import EncoderConfig, EncoderMLM, ResNet50

MODELS = ["resnet", "encoder"]


def _model(name, device="cpu"):
    torch.manual_seed(0)
    with torch.device(device):
        if name == "resnet":
            return ResNet50.tiny(), torch.randn(2, 3, 64, 64).contiguous(memory_format=torch.channels_last)
        cfg = EncoderConfig.tiny()
        return EncoderMLM(cfg), torch.randint(0, cfg.vocab, (2, cfg.seq_len))


def _capture(how, model, x):
    if how == "fx":
        return torch.fx.symbolic_trace(model, concrete_args={"labels": None})(x, None)
    if how == "script":
        return torch.jit.script(model)(x)
    if how == "trace":
        return torch.jit.trace(model, (x,), check_trace=False)(x)
    if how == "make_fx":
        return make_fx(model)(x)(x)
    if how == "compile":
        torch._dynamo.reset()
        return torch.compile(model, fullgraph=True, backend="eager")(x)
    assert how == "export"
    return torch.export.export(model, (x,)).module()(x)


HOW = ["fx", "script", "trace", "make_fx", "compile", "export"]


@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("how", HOW)
def test_captured_models_give_what_the_model_gives(name, how):
    model, x = _model(name)
    model.eval()
    torch.testing.assert_close(_capture(how, model, x), model(x), rtol=1e-5, atol=1e-5)


def test_a_traced_resnet_names_its_modules():
    graph = torch.fx.symbolic_trace(ResNet50.tiny(), concrete_args={"labels": None}).graph
    called = {n.target for n in graph.nodes if n.op == "call_module"}
    assert {"conv1", "bn1", "maxpool", "layer1.0.bn3", "layer2.0.downsample.1", "fc"} <= called


@pytest.mark.parametrize("name", MODELS)
def test_fake_gpu_tensors(name):
    """The shapes of a training step's forward, without a GPU: nothing may ask for an address."""
    with FakeTensorMode():
        model, x = _model(name, "cuda")
        labels = torch.zeros(2, dtype=torch.long, device="cuda") if name == "resnet" else None
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = model(x, labels)
    assert out.requires_grad and out.device.type == "cuda" and out.shape == (() if name == "resnet" else (2, 32, 1000))


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


@pytest.fixture
def _every_size(monkeypatch):
    """Below these sizes the modules are called in any case."""
    import sys

    import fairring_b200.models  # noqa: F401

    for module, name in (("ops.layernorm", "_PAIR_FROM"), ("ops.embedding", "_PAD_FROM"), ("ops.linear", "_FUSE_FROM"),
                         ("ops.stem", "_FOLD_FROM"), ("ops._plain", "FUSE_FROM")):
        monkeypatch.setattr(sys.modules["fairring_b200." + module], name, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("how", HOW)
def test_captured_on_the_gpu(name, how, _every_size):
    """In training mode under autocast, where the package's own ops would run."""
    _need_gpu()
    model, x = _model(name, "cuda")
    model.train()
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=how not in ("trace", "make_fx")):
        got, want = _capture(how, model, x), model(x)
    assert float((got - want).norm()) <= 0.03 * float(want.norm())  # other kernels, in bf16


@pytest.mark.gpu
@pytest.mark.parametrize("name", MODELS)
def test_transforms_and_modes_on_the_gpu(name, _every_size):
    _need_gpu()
    model, x = _model(name, "cuda")
    model.eval()  # running statistics are not written under a transform
    params = {k: v.detach() for k, v in model.named_parameters()}
    loss = lambda p: functional_call(model, p, (x,)).float().square().mean()  # noqa: E731
    grads = grad(loss)(params)
    want = torch.autograd.grad(loss(dict(model.named_parameters())), list(model.parameters()))
    for g, w in zip(grads.values(), want):
        torch.testing.assert_close(g, w, rtol=1e-3, atol=1e-4 * float(w.abs().max()))
    if name == "resnet":  # torch's attention has no forward-mode derivative
        along = {k: torch.randn_like(v) for k, v in params.items()}
        slope = sum(float((along[k] * grads[k]).sum()) for k in params)
        got = float(jvp(loss, (params,), (along,))[1])
        assert abs(got - slope) <= 1e-3 * sum(float((along[k] * grads[k]).abs().sum()) for k in params) ** 0.5 + 1e-3 * abs(slope)
    model.train()
    with FlopCounterMode(display=False) as counted, torch.autocast("cuda", dtype=torch.bfloat16):
        model(x)
    assert counted.get_total_flops() > 0
    with torch.inference_mode(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert bool(model(x).isfinite().all())
