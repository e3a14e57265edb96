"""What a user of this library has it do on one GPU, as cases that can be timed.

A case is a dict of plain values; :func:`prepare` makes what a program holds before the call,
:func:`run` is one pass through the public entry points, :func:`work` says what a pass cannot do
without and :func:`tolerance` how far another correct implementation may be off.  Seven kinds:

``static``    ``fairring_allreduce_f32_noalloc``: 2 to 8 buffers of one device, up to 4096 floats
``norm``      ``FusedLayerNorm`` forward and backward
``residual``  ``add_layer_norm`` forward and backward (residual stream fp32, branch bf16 or fp32)
``loss``      ``fused_cross_entropy`` forward and backward on the logits of a language-model head
``adamw``     ``FlatAdamW``: gradient norm and step over a flat buffer
``decoder``, ``encoder``, ``resnet``  one data-parallel training step of the three workloads, with
              the wrapper, the optimizer and the options that ``bench.py`` and ``train/run.py`` use

All-reduce between GPUs needs several of them and is timed by ``fairring_b200.bench.sweep``.
"""

import ctypes
import math
import os

import torch
import torch.distributed as dist
import torch.nn.functional as F

import fairring_b200
from fairring_b200.models import DecoderConfig, DecoderLM, EncoderConfig, EncoderMLM, ResNet50, mask_tokens
from fairring_b200.ops import FlatAdamW, FusedLayerNorm, add_layer_norm, fused_cross_entropy
from fairring_b200.parallel import FlatDataParallel

DEVICE = "cuda"
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
HEAD_WIDTH = 128  # width of the hidden state behind the logits of the `loss` cases


# ---- the cases --------------------------------------------------------------------------------
def listed():
    return [
        # The smallest reductions: a plugin that sums two short vectors between kernels of its
        # host; the whole call is launch latency.
        {"name": "static_2x1000", "kind": "static", "world": 2, "numel": 1000},
        # The largest reduction that this entry point takes.
        {"name": "static_8x4096", "kind": "static", "world": 8, "numel": 4096},
        # LayerNorm of bf16 activations at a row count and a row length that divide into nothing
        # (both from the tests).
        {"name": "norm_777x4104", "kind": "norm", "rows": 777, "cols": 4104, "x": "bf16", "autocast": True},
        # The decoder's hot normalisation: 8 x 1024 tokens of width 2048, bf16 branch, autocast.
        {"name": "residual_8192x2048", "kind": "residual", "rows": 8192, "cols": 2048, "branch": "bf16"},
        # The decoder's loss: 8 x 1024 rows over a vocabulary of 51200.
        {"name": "loss_8192x51200", "kind": "loss", "rows": 8192, "vocab": 51200, "logits": "bf16", "ignored": 0.0},
        # The masked-LM loss: 15 % of 16 x 512 positions over a vocabulary of 50265, an odd number.
        {"name": "loss_1229x50265", "kind": "loss", "rows": 1229, "vocab": 50265, "logits": "bf16", "ignored": 0.0},
        # The optimizer over as many parameters as ResNet-50 has, with the gradient norm that a
        # training loop logs.
        {"name": "adamw_25m", "kind": "adamw", "numel": 25_557_032, "shadow": False},
        # The small test model (2 layers of width 128): host work and launches.
        {"name": "decoder_tiny", "kind": "decoder", "layers": 2, "d_model": 128, "heads": 4, "vocab": 1024,
         "seq": 64, "batch": 4, "micro": 1},
        # Two layers of the benchmark's decoder, one sequence at a time, two micro-batches per step
        # (gradient accumulation under no_sync).
        {"name": "decoder_2l_accum", "kind": "decoder", "layers": 2, "d_model": 2048, "heads": 16, "vocab": 51200,
         "seq": 1024, "batch": 1, "micro": 2},
        # The benchmark's decoder as bench.py trains it: the largest case.
        {"name": "decoder_1p4b", "kind": "decoder", "layers": 26, "d_model": 2048, "heads": 16, "vocab": 51200,
         "seq": 1024, "batch": 8, "micro": 1},
        # The 1.3 B masked-LM encoder as train/run.py trains it.
        {"name": "encoder_1p3b", "kind": "encoder", "layers": 24, "d_model": 2048, "heads": 32, "vocab": 50265,
         "seq": 512, "batch": 16},
        # ResNet-50 as train/run.py trains it (channels-last, bf16 autocast, fp16 wire).
        {"name": "resnet50_b256", "kind": "resnet", "batch": 256, "size": 224},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "norm", "residual", "loss", "adamw", "decoder", "encoder", "resnet"])
    if kind == "static":
        return {"kind": kind, "world": rng.randint(2, 8), "numel": _log_uniform(rng, 1, 4096)}
    if kind == "norm":
        x, autocast = rng.choice([("fp32", True), ("fp32", False), ("bf16", True)])
        return {"kind": kind, "rows": _log_uniform(rng, 16, 16384), "cols": 8 * _log_uniform(rng, 16, 1024),
                "x": x, "autocast": autocast}
    if kind == "residual":
        return {"kind": kind, "rows": _log_uniform(rng, 16, 16384), "cols": 8 * _log_uniform(rng, 16, 1024),
                "branch": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "loss":
        return {"kind": kind, "rows": _log_uniform(rng, 64, 8192), "vocab": _log_uniform(rng, 1000, 51200),
                "logits": rng.choice(["bf16", "bf16", "fp32"]), "ignored": rng.choice([0.0, 0.15])}
    if kind == "adamw":
        return {"kind": kind, "numel": _log_uniform(rng, 10_000, 300_000_000), "shadow": rng.random() < 0.5}
    if kind == "decoder":
        heads = rng.choice([2, 4, 8, 16])
        return {"kind": kind, "layers": rng.randint(1, 6), "d_model": heads * rng.choice([32, 64, 128]),
                "heads": heads, "vocab": 8 * _log_uniform(rng, 125, 6400), "seq": _log_uniform(rng, 32, 1024),
                "batch": rng.randint(1, 8), "micro": rng.choice([1, 1, 2])}
    if kind == "encoder":
        heads = rng.choice([2, 4, 8, 16])
        return {"kind": kind, "layers": rng.randint(1, 6), "d_model": heads * rng.choice([32, 64]),
                "heads": heads, "vocab": _log_uniform(rng, 1000, 50265), "seq": _log_uniform(rng, 32, 512),
                "batch": rng.randint(1, 16)}
    return {"kind": kind, "batch": _log_uniform(rng, 16, 128), "size": 32 * rng.randint(3, 7)}


# ---- one GPU, one process ------------------------------------------------------------------------
def _process_group():
    """The "fairring" group of a single rank, created once per process as a training script does."""
    if not dist.is_initialized():
        os.environ.setdefault("FAIRRING_TOTAL_MEMORY", str(256 << 20))
        dist.init_process_group("fairring", store=dist.HashStore(), rank=0, world_size=1)


def _static_entry():
    lib = ctypes.CDLL(os.path.join(os.path.dirname(fairring_b200.__file__), "_C.so"))
    fn = lib.fairring_allreduce_f32_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p,
                   ctypes.c_int, ctypes.c_char_p, ctypes.c_ulong]
    return fn


# ---- static ----------------------------------------------------------------------------------
def _prepare_static(case, gen):
    contributions = torch.randn(case["world"], case["numel"], device=DEVICE, generator=gen)
    buffers = torch.empty_like(contributions)
    pointers = (ctypes.c_void_p * case["world"])(*[b.data_ptr() for b in buffers])
    return {"fn": _static_entry(), "contributions": contributions, "buffers": buffers, "pointers": pointers}


def _run_static(case, s):
    s["buffers"].copy_(s["contributions"])  # each pass has something new to sum
    rc = s["fn"](s["pointers"], case["world"], case["numel"],
                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), 0, None, 0)
    if rc != 0:
        raise RuntimeError(f"fairring_allreduce_f32_noalloc returned {rc}")
    return s["buffers"]


# ---- norm, residual ----------------------------------------------------------------------------
def _norm_module(cols, gen):
    norm = FusedLayerNorm(cols, device=DEVICE)
    with torch.no_grad():
        norm.weight.normal_(1.0, 0.2, generator=gen)
        norm.bias.normal_(0.0, 0.2, generator=gen)
    return norm


def _prepare_norm(case, gen):
    shape = (case["rows"], case["cols"])
    x = (torch.randn(shape, device=DEVICE, generator=gen) * 2 + 0.5).to(DTYPES[case["x"]]).requires_grad_(True)
    out = torch.bfloat16 if case["autocast"] else x.dtype
    dy = torch.randn(shape, device=DEVICE, generator=gen).to(out)
    return {"norm": _norm_module(case["cols"], gen), "x": x, "dy": dy}


def _run_norm(case, s):
    norm = s["norm"]
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["autocast"]):
        y = norm(s["x"])
    return [y, *torch.autograd.grad(y, [s["x"], norm.weight, norm.bias], s["dy"])]


def _prepare_residual(case, gen):
    shape = (case["rows"], case["cols"])
    branch_dtype = DTYPES[case["branch"]]
    return {"norm": _norm_module(case["cols"], gen),
            "x": torch.randn(shape, device=DEVICE, generator=gen).requires_grad_(True),
            "branch": torch.randn(shape, device=DEVICE, generator=gen).to(branch_dtype).requires_grad_(True),
            "dstream": torch.randn(shape, device=DEVICE, generator=gen),
            "dy": torch.randn(shape, device=DEVICE, generator=gen).to(branch_dtype)}


def _run_residual(case, s):
    norm = s["norm"]
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["branch"] == "bf16"):
        stream, y = add_layer_norm(norm, s["x"], s["branch"])
    grads = torch.autograd.grad([stream, y], [s["x"], s["branch"], norm.weight, norm.bias], [s["dstream"], s["dy"]])
    return [stream, y, *grads]


# ---- loss --------------------------------------------------------------------------------------
def _prepare_loss(case, gen):
    rows, vocab = case["rows"], case["vocab"]
    hidden = torch.randn(rows, HEAD_WIDTH, device=DEVICE, generator=gen).to(torch.bfloat16)
    head = torch.randn(vocab, HEAD_WIDTH, device=DEVICE, generator=gen) * (2.0 / math.sqrt(HEAD_WIDTH))
    targets = torch.randint(0, vocab, (rows,), device=DEVICE, generator=gen)
    if case["ignored"]:
        targets[torch.rand(rows, device=DEVICE, generator=gen) < case["ignored"]] = -100
    return {"hidden": hidden, "head": head.to(torch.bfloat16).requires_grad_(True), "targets": targets}


def _run_loss(case, s):
    logits = F.linear(s["hidden"], s["head"])  # the loss consumes its logits: they come out of an op
    if case["logits"] == "fp32":
        logits = logits.float()
    loss = fused_cross_entropy(logits, s["targets"])
    return [loss, torch.autograd.grad(loss, logits)[0]]


# ---- adamw --------------------------------------------------------------------------------------
def _prepare_adamw(case, gen):
    n = case["numel"]
    param = torch.randn(n, device=DEVICE, generator=gen).mul_(0.02)
    grad = torch.randn(n, device=DEVICE, generator=gen).mul_(1e-3)
    shadow = param.to(torch.bfloat16) if case["shadow"] else None
    return {"opt": FlatAdamW(param, grad, lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1, shadow=shadow)}


def _run_adamw(case, s):
    opt = s["opt"]
    norm = opt.grad_norm()
    opt.step()
    return [norm, opt.param, opt.exp_avg, opt.exp_avg_sq, opt.shadow]


# ---- training steps ------------------------------------------------------------------------------
class _Training:
    """The wrapper, its optimizer and one batch.  The wrapper and its parameters hold each other
    through gradient hooks, which the garbage collector cannot follow: a program that makes several
    wrappers takes each apart when it is done with it."""

    def __init__(self, ddp, opt, **batch):
        self.ddp, self.opt, self.batch = ddp, opt, batch

    def __del__(self):
        self.ddp.__dict__.clear()


def _prepare_decoder(case, gen):
    cfg = DecoderConfig(n_layer=case["layers"], d_model=case["d_model"], n_head=case["heads"],
                        d_ff=4 * case["d_model"], vocab=case["vocab"], seq_len=case["seq"])
    with torch.device(DEVICE):
        model = DecoderLM(cfg)
    ddp = FlatDataParallel(model, bf16_shadow=True)
    opt = FlatAdamW(ddp.flat_param, ddp.flat_grad, lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1,
                    shadow=ddp.flat_shadow, overlap=ddp)
    tokens = torch.randint(0, cfg.vocab, (case["micro"], case["batch"], cfg.seq_len + 1), device=DEVICE, generator=gen)
    return {"training": _Training(ddp, opt, tokens=tokens)}


def _run_decoder(case, s):
    ddp, opt, tokens = s["training"].ddp, s["training"].opt, s["training"].batch["tokens"]

    def micro(block):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = ddp(block[:, :-1], block[:, 1:])
        loss.backward()
        return loss.detach()

    losses = []
    for block in tokens[:-1]:
        with ddp.no_sync():
            losses.append(micro(block))
    losses.append(micro(tokens[-1]))
    opt.step()
    opt.zero_grad(set_to_none=True)
    return [*losses, ddp.flat_grad, ddp.flat_param]


def _prepare_encoder(case, gen):
    cfg = EncoderConfig(n_layer=case["layers"], d_model=case["d_model"], n_head=case["heads"],
                        d_ff=4 * case["d_model"], vocab=case["vocab"], seq_len=case["seq"])
    with torch.device(DEVICE):
        model = EncoderMLM(cfg)
    ddp = FlatDataParallel(model)
    opt = FlatAdamW(ddp.flat_param, ddp.flat_grad, lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1)
    host = torch.Generator().manual_seed(gen.initial_seed())
    tokens = torch.randint(1, cfg.vocab, (case["batch"], cfg.seq_len), generator=host)
    tokens, labels = mask_tokens(tokens, cfg, host)
    labels[0, 0] = 1  # never a batch without a single masked position
    return {"training": _Training(ddp, opt, x=tokens.to(DEVICE), y=labels.to(DEVICE))}


def _prepare_resnet(case, gen):
    with torch.device(DEVICE):
        model = ResNet50()
    ddp = FlatDataParallel(model.to(memory_format=torch.channels_last), wire_dtype=torch.float16)
    opt = FlatAdamW(ddp.flat_param, ddp.flat_grad, lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1)
    images = torch.randn(case["batch"], 3, case["size"], case["size"], device=DEVICE, generator=gen)
    labels = torch.randint(0, 1000, (case["batch"],), device=DEVICE, generator=gen)
    return {"training": _Training(ddp, opt, x=images.contiguous(memory_format=torch.channels_last), y=labels)}


def _step(training):
    ddp, opt, batch = training.ddp, training.opt, training.batch
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = ddp(batch["x"], batch["y"])
    loss.backward()
    opt.step()
    opt.zero_grad(set_to_none=True)
    return loss.detach()


def _run_encoder(case, s):
    t = s["training"]
    return [_step(t), t.ddp.flat_grad, t.ddp.flat_param]


def _run_resnet(case, s):
    """The loss, the updated weights and the running statistics at the end of three stages.  Not the
    gradients: at random weights those of a 50-layer network with batch norm are as good as
    unrelated (relative difference 1.1) between two orders of the same bf16 sums."""
    t = s["training"]
    loss = _step(t)
    net = t.ddp.module
    norms = [net.bn1, net.layer1[-1].bn3, net.layer2[-1].bn3, net.layer3[-1].bn3]
    return [loss, t.ddp.flat_param, *[b for m in norms for b in (m.running_mean, m.running_var)]]


_PREPARE = {"static": _prepare_static, "norm": _prepare_norm, "residual": _prepare_residual, "loss": _prepare_loss,
            "adamw": _prepare_adamw, "decoder": _prepare_decoder, "encoder": _prepare_encoder,
            "resnet": _prepare_resnet}
_RUN = {"static": _run_static, "norm": _run_norm, "residual": _run_residual, "loss": _run_loss,
        "adamw": _run_adamw, "decoder": _run_decoder, "encoder": _run_encoder, "resnet": _run_resnet}


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    torch.manual_seed(seed)  # initial weights
    if case["kind"] in ("decoder", "encoder", "resnet"):
        _process_group()
    return {"case": case, **_PREPARE[case["kind"]](case, gen)}


def run(state):
    case = state["case"]
    return _RUN[case["kind"]](case, state)


# ---- what a pass cannot do without ---------------------------------------------------------------
def _transformer_work(layers, d, vocab, rows, seq, head_rows, causal, shadow):
    """Forward and backward of `rows` tokens: matrix products, attention, the head, the optimizer."""
    weights = layers * 12 * d * d
    params = weights + layers * 13 * d + (vocab + seq) * d + 2 * d
    flops = 6 * weights * rows + 6 * vocab * d * head_rows
    flops += layers * 12 * rows * seq * d * (0.5 if causal else 1.0)
    # parameters and both moments read and written, the gradient written; the bf16 copy with them
    return {"bytes": params * (28 + (2 if shadow else 0)), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "static":
        return {"bytes": 2 * 4 * case["world"] * case["numel"], "flops": (case["world"] - 1) * case["numel"]}
    if kind == "norm":
        n, x = case["rows"] * case["cols"], 2 if case["x"] == "bf16" else 4
        y = 2 if case["autocast"] else x
        # forward: x in, y out; backward: dy and x in, dx out
        return {"bytes": n * (3 * x + 2 * y), "flops": 20 * n}
    if kind == "residual":
        n, b = case["rows"] * case["cols"], 2 if case["branch"] == "bf16" else 4
        # forward: x and branch in, stream and y out; backward: dy, stream and its gradient in,
        # the gradients of x and of the branch out (one and the same in fp32)
        return {"bytes": n * ((4 + b + 4 + b) + (b + 4 + 4) + 4 + (b if b == 2 else 0)), "flops": 22 * n}
    if kind == "loss":
        n, b = case["rows"] * case["vocab"], 2 if case["logits"] == "bf16" else 4
        # the logits come out of the head once; the loss reads them, the gradient reads and writes them
        return {"bytes": 4 * b * n, "flops": n * (2 * HEAD_WIDTH + 8)}
    if kind == "adamw":
        return {"bytes": case["numel"] * (28 + (2 if case["shadow"] else 0)), "flops": 15 * case["numel"]}
    if kind == "decoder":
        rows = case["micro"] * case["batch"] * case["seq"]
        return _transformer_work(case["layers"], case["d_model"], case["vocab"], rows, case["seq"], rows, True, True)
    if kind == "encoder":
        rows = case["batch"] * case["seq"]
        return _transformer_work(case["layers"], case["d_model"], case["vocab"], rows, case["seq"], int(0.15 * rows) + 1,
                                 False, False)
    scale = (case["size"] / 224.0) ** 2
    return {"bytes": 25_557_032 * 28 + case["batch"] * 3 * case["size"] ** 2 * 4,
            "flops": case["batch"] * scale * 3 * 2 * 4.09e9}


def tolerance(case):
    """Four times what was seen against the same values in 64 bits (the kernels by themselves) or, for
    training steps, against the same step from other kernels (plain LayerNorm, loss and residual
    adds; another attention; NCHW instead of channels-last)."""
    kind = case["kind"]
    if kind == "static":  # seen: 5.8e-8, largest 3.1e-7
        return {"rel": 2.5e-7, "max": 1.3e-6}
    if kind in ("norm", "residual"):
        narrow = case["autocast"] if kind == "norm" else case["branch"] == "bf16"
        # bf16 results: 1.7e-3, largest 3.9e-3 (half a step of the format); fp32: 1.4e-7 and 5.1e-7
        return {"rel": 7e-3, "max": 1.6e-2} if narrow else {"rel": 6e-7, "max": 2.1e-6}
    if kind == "loss":  # bf16 gradients: 1.4e-3, largest 3.9e-3; fp32: 8e-8 and 1.0e-6
        return {"rel": 6e-3, "max": 1.6e-2} if case["logits"] == "bf16" else {"rel": 3.2e-7, "max": 4e-6}
    if kind == "adamw":  # fp32: 2.4e-7, largest 3.4e-7; the bf16 copy: 1.7e-3 and 3.9e-3
        return {"rel": 7e-3, "max": 1.6e-2} if case["shadow"] else {"rel": 1e-6, "max": 1.4e-6}
    if kind in ("decoder", "encoder"):  # gradients under bf16 autocast: 8.4e-3 (24 layers: 1.4e-2), largest 0.74
        return {"rel": 0.03, "max": 0.99}
    # loss 3.6e-3, weights 2.0e-3, running statistics 4.1e-3
    return {"rel": 1.6e-2, "max": 0.2}
