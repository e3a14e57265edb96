"""The post-LayerNorm pair and the encoder on it."""

import sys

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _small_sizes_too(monkeypatch):
    """Below these sizes the modules are called; the tests are about what runs above."""
    import fairring_b200.ops  # noqa: F401

    monkeypatch.setattr(sys.modules["fairring_b200.ops.layernorm"], "_PAIR_FROM", 0)
    monkeypatch.setattr(sys.modules["fairring_b200.ops.embedding"], "_PAD_FROM", 0)
    monkeypatch.setattr(sys.modules["fairring_b200.ops._plain"], "FUSE_FROM", 0)
    monkeypatch.setattr(sys.modules["fairring_b200.ops.linear"], "_FUSE_FROM", 0)


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


@pytest.mark.parametrize("cols", [8, 264, 2048, 8192])
@pytest.mark.parametrize("use", ["both", "fp32", "low"])
@pytest.mark.parametrize("branch_dtype", [torch.bfloat16, torch.float32])
def test_pair_against_fp64(cols, use, branch_dtype):
    _need_gpu()
    from fairring_b200.ops import add_layer_norm_pair

    gen = torch.Generator(device="cuda").manual_seed(cols)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    rows = 301
    norm = nn.LayerNorm(cols, device="cuda")
    with torch.no_grad():
        norm.weight.normal_(1.0, 0.2, generator=gen)
        norm.bias.normal_(0.0, 0.2, generator=gen)
    x, br = rand(rows, cols).requires_grad_(True), rand(rows, cols).to(branch_dtype).requires_grad_(True)
    d32, dlow = rand(rows, cols), rand(rows, cols).bfloat16()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y, low = add_layer_norm_pair(norm, x, br)
    assert y.dtype == torch.float32 and low.dtype == torch.bfloat16
    outs = {"both": ([y, low], [d32, dlow]), "fp32": ([y], [d32]), "low": ([low], [dlow])}[use]
    grads = torch.autograd.grad(outs[0], [x, br, norm.weight, norm.bias], outs[1])
    leaves = [t.detach().double().requires_grad_(True) for t in (x, br, norm.weight, norm.bias)]
    want = F.layer_norm(leaves[0] + leaves[1], (cols,), leaves[2], leaves[3], norm.eps)
    wants = torch.autograd.grad(want, leaves, sum(d.double() for d in outs[1]))
    assert float((y.double() - want).abs().max()) < 4e-6 * float(want.detach().abs().max())
    assert torch.equal(low, y.bfloat16())
    for got, ref in zip(grads, wants):
        eps = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -21
        assert ((got.double() - ref).abs() <= eps * ref.abs() + 1e-5 * max(1.0, float(ref.abs().max()))).all()


@pytest.mark.parametrize("cols", [128, 2048, 4104, 8192])
def test_a_mean_far_from_zero_keeps_the_variance(cols):
    _need_gpu()
    from fairring_b200.ops import add_layer_norm_pair

    x = torch.randn(64, cols, device="cuda") + 1000
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y, _ = add_layer_norm_pair(nn.LayerNorm(cols, device="cuda"), x, torch.zeros_like(x))
    # x - mean is exact to half a step of fp32 at 1000, 3e-5
    assert float((y.double() - F.layer_norm(x.double(), (cols,))).abs().max()) < 2e-4


@pytest.mark.parametrize("branch_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("use", ["both", "fp32", "low"])
def test_pair_second_derivative(use, branch_dtype):
    _need_gpu()
    from fairring_b200.ops import add_layer_norm_pair

    gen = torch.Generator(device="cuda").manual_seed(11)
    x0, br0 = torch.randn(12, 24, device="cuda", generator=gen), torch.randn(12, 24, device="cuda", generator=gen)
    got = []
    for fused in (True, False):
        norm = nn.LayerNorm(24, device="cuda")
        x, br = x0.clone().requires_grad_(True), br0.to(branch_dtype).requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            if fused:
                y, low = add_layer_norm_pair(norm, x, br)
                assert type(y.grad_fn).__name__ == "_AddLayerNormPairFnBackward"
            else:
                y = norm(x + br)
                low = y.bfloat16()
        out = (0.0 if use == "low" else (y ** 3).sum()) + (0.0 if use == "fp32" else (low.float() ** 3).sum())
        leaves = [x, br, norm.weight, norm.bias]
        first = torch.autograd.grad(out, leaves, create_graph=True)
        assert all(g.requires_grad for g in first)
        got.append([*first, *torch.autograd.grad(sum((g.float() ** 2).sum() for g in first), leaves)])
    rtol = 2.0 ** -5 if branch_dtype == torch.bfloat16 or use != "fp32" else 1e-3  # up to four roundings to bf16
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=rtol, atol=rtol * float(b.detach().abs().max()))


@pytest.mark.parametrize("vocab", [1000, 1001, 1007])
@pytest.mark.parametrize("rows", [37, 0])
def test_padded_head_matches_torch(vocab, rows):
    _need_gpu()
    from fairring_b200.ops import cross_entropy_keeping_logits, tied_embedding, vocab_logits

    torch.manual_seed(vocab)
    tok, pos = nn.Embedding(vocab, 64, device="cuda"), nn.Embedding(8, 64, device="cuda")
    b = torch.randn(vocab, device="cuda").requires_grad_(True)
    h = torch.randn(rows, 64, device="cuda").requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda")
    tokens = torch.randint(0, vocab, (2, 8), device="cuda")
    got = []
    with torch.autocast("cuda", dtype=torch.bfloat16):
        x, table = tied_embedding(tok, pos, tokens, pad_rows=True)
        assert table.shape[0] == (vocab + 7) // 8 * 8
        loss = cross_entropy_keeping_logits(vocab_logits(h, table, b), t)
        got.append([loss, *torch.autograd.grad(loss + x.sum(), [h, tok.weight, b])])
        x = tok(tokens) + pos(torch.arange(8, device="cuda"))
        loss = F.cross_entropy(F.linear(h, tok.weight, b).float(), t)
        got.append([loss, *torch.autograd.grad(loss + x.sum(), [h, tok.weight, b])])
    for a, r in zip(*got):
        assert a.dtype == r.dtype and a.shape == r.shape
        scale = float(r.detach().nan_to_num().abs().max()) if r.numel() else 0.0  # no row: a loss of NaN
        torch.testing.assert_close(a, r, rtol=2.0 ** -6, atol=2.0 ** -7 * scale, equal_nan=True)


FUSED = {"_TiedEmbeddingFnBackward", "_AddLayerNormPairFnBackward", "_BiasGradFnBackward", "_GeluFnBackward",
         "_PaddedHeadFnBackward"}


def _nodes(loss):
    """The names of all autograd nodes behind `loss`."""
    seen, todo, names = set(), [loss.grad_fn], set()
    while todo:
        fn = todo.pop()
        if fn is not None and fn not in seen:
            seen.add(fn)
            names.add(type(fn).__name__)
            todo += [f for f, _ in fn.next_functions]
    return names


def test_encoder_matches_its_plain_layers():
    _need_gpu()
    from fairring_b200.models import EncoderConfig, EncoderMLM, mask_tokens

    torch.manual_seed(0)
    cfg = EncoderConfig(n_layer=2, d_model=128, n_head=4, d_ff=512, vocab=1001, seq_len=32)
    model = EncoderMLM(cfg).cuda()
    gen = torch.Generator().manual_seed(1)
    tokens, labels = mask_tokens(torch.randint(1, cfg.vocab, (4, 32), generator=gen), cfg, gen)
    tokens, labels = tokens.cuda(), labels.cuda()
    got = []
    for hooked in (False, True):
        if hooked:  # a hook makes each module be called by itself
            for m in model.modules():
                m.register_forward_hook(lambda *a: None)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = model(tokens, labels)
        assert _nodes(loss) >= FUSED if not hooked else not _nodes(loss) & FUSED
        got.append([loss, *torch.autograd.grad(loss, list(model.parameters()))])
    assert abs(float(got[0][0]) - float(got[1][0])) < 2e-3 * float(got[1][0])
    for a, r in zip(got[0][1:], got[1][1:]):
        assert float((a - r).norm()) <= 0.03 * float(r.norm()) + 1e-6
