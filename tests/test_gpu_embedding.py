"""The tied embedding against torch's modules."""

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


# one column group, a ragged block, a second block of columns; one sequence, fewer tokens than positions,
# a token that fills most of the batch
@pytest.mark.parametrize("d", [8, 264, 1032, 2048])
@pytest.mark.parametrize("batch,seq,positions", [(1, 1, 1), (5, 33, 40), (9, 64, 64)])
@pytest.mark.parametrize("use", ["both", "lookup", "projection"])
def test_matches_torch(d, batch, seq, positions, use):
    _need_gpu()
    from fairring_b200.ops import tied_embedding

    gen = torch.Generator(device="cuda").manual_seed(d + seq)
    tok, pos = nn.Embedding(101, d, device="cuda"), nn.Embedding(positions, d, device="cuda")
    tokens = torch.randint(0, 101, (batch, seq), device="cuda", generator=gen)
    tokens[:, ::2] = 7
    h = torch.randn(50, d, device="cuda", generator=gen).bfloat16()
    dx = torch.randn(batch, seq, d, device="cuda", generator=gen)
    dl = torch.randn(50, 101, device="cuda", generator=gen).bfloat16()
    got = []
    for fused in (True, False):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            if fused:
                x, table = tied_embedding(tok, pos, tokens)
                assert table.dtype == torch.bfloat16
            else:
                x, table = tok(tokens) + pos(torch.arange(seq, device="cuda")), tok.weight
            logits = F.linear(h, table)
        outs = {"both": ([x, logits], [dx, dl]), "lookup": ([x], [dx]), "projection": ([logits], [dl])}[use]
        params = [tok.weight, pos.weight] if use != "projection" else [tok.weight]
        got.append([x, logits, *torch.autograd.grad(outs[0], params, outs[1])])
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    for a, b in zip(got[0][2:], got[1][2:]):  # sums of up to batch * seq / 2 rows in another order
        assert a.dtype == b.dtype == torch.float32
        assert float((a - b).abs().max()) <= 2e-6 * (batch * seq) ** 0.5 * max(1.0, float(b.abs().max()))


# less than one round of 2048 tokens, a ragged second and third; tokens of a few occurrences, lists long enough
# to take a frequent token out, and a batch of nothing else
@pytest.mark.parametrize("d", [8, 136, 2048])
@pytest.mark.parametrize("batch,seq", [(1, 7), (3, 700), (5, 1001)])
@pytest.mark.parametrize("mix", ["spread", "frequent", "one"])
def test_the_gradient_repeats_itself(d, batch, seq, mix):
    _need_gpu()
    from fairring_b200 import _C

    vocab, n = 613, batch * seq
    gen = torch.Generator(device="cuda").manual_seed(d + n)
    tokens = torch.randint(0, vocab, (batch, seq), device="cuda", generator=gen)
    if mix == "frequent":
        tokens[torch.rand(batch, seq, device="cuda", generator=gen) < 0.4] = 612
        tokens[:, ::9] = 3
    elif mix == "one":
        tokens[:] = 5
    dx = torch.randn(batch, seq, d, device="cuda", generator=gen)
    dlow = torch.randn(vocab, d, device="cuda", generator=gen).bfloat16()
    dtable, dpos = _C.embed_bwd(dx, dlow, tokens, vocab, seq + 2, d)
    rows = dx.view(n, d).double()
    want = dlow.double().index_add_(0, tokens.view(-1), rows)
    most = dlow.double().abs().index_add_(0, tokens.view(-1), rows.abs())  # a rounding for each term at the most
    times = torch.bincount(tokens.view(-1), minlength=vocab).view(-1, 1) + 1
    assert ((dtable.double() - want).abs() <= 2.0 ** -24 * times * most).all()
    assert ((dpos[:seq].double() - dx.double().sum(0)).abs() <= 2.0 ** -24 * batch * dx.double().abs().sum(0)).all()
    assert not dpos[seq:].any()
    for _ in range(3):
        again = _C.embed_bwd(dx, dlow, tokens, vocab, seq + 2, d)
        assert torch.equal(again[0], dtable) and torch.equal(again[1], dpos)


def test_no_tokens():
    _need_gpu()
    from fairring_b200 import _C

    junk = [torch.full((4, 8), 7.0, device="cuda") for _ in range(8)]  # what the allocator hands out next
    del junk
    dtable, dpos = _C.embed_bwd(torch.empty(0, 4, 8, device="cuda"), None, torch.empty(0, 4, dtype=torch.long, device="cuda"),
                                5, 4, 8)
    assert not dtable.any() and not dpos.any()


def test_calls_the_modules_where_they_cannot_be_skipped():
    _need_gpu()
    from fairring_b200.ops import tied_embedding

    pos, tokens = nn.Embedding(4, 8, device="cuda"), torch.tensor([[0, 1, 2]], device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        for tok in (nn.Embedding(5, 8, device="cuda", padding_idx=0), nn.Embedding(5, 8, device="cuda", max_norm=1.0)):
            assert tied_embedding(tok, pos, tokens)[1] is tok.weight
        tok = nn.Embedding(5, 8, device="cuda")
        seen = []
        handle = tok.register_forward_hook(lambda *a: seen.append(1))
        tied_embedding(tok, pos, tokens)
        handle.remove()
        assert seen == [1]
        assert tied_embedding(tok, pos, tokens)[1].dtype == torch.bfloat16
    assert tied_embedding(tok, pos, tokens)[1] is tok.weight  # no autocast
