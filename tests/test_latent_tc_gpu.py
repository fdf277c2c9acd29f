"""Attention over a latent on tcgen05 at the edges of its tiles, against the same attention in float64: contexts around multiples of
32 and 64 keys, portions around multiples of 128 (token, head) rows, head counts that put rows of one token into two tiles, latents of one
piece of 256 columns and of two, part-filled blocks of 64 columns, pages shorter and longer than a tile of keys, sinks, scores large
enough to move the maximum late.  The cache holds NaN behind every context.  Bound: sums of bfloat16 operands in float32, weights
in two bfloat16 halves (2^-16), the result rounded to bfloat16 (2^-8, twice for the order of rounding)."""

import pytest
import torch

from clockwork_b200 import ops
from clockwork_b200.ops import latent as latent_ops
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu


class Holder:
    pass


@pytest.mark.parametrize("heads, rank, rot, page, sharp", [(16, 512, 64, 16, 1.0), (5, 272, 16, 8, 1.0), (3, 64, 32, 32, 6.0), (16, 256, 0, 64, 1.0),
                                                           (130, 48, 16, 16, 3.0)])
@pytest.mark.parametrize("sink", [False, True])
def test_portions(monkeypatch, heads, rank, rot, page, sharp, sink):
    g = torch.Generator().manual_seed(heads + rank)
    D, scale = rank + rot, (rank + rot) ** -0.5
    behind, new = [0, 31, 100, 1, 500, 64], [8, 1, 29, 31, 13, 64]
    n, seqs = sum(new) + 3, len(new)
    ctx_lens = [b + q for b, q in zip(behind, new)]
    pages = [-(-c // page) for c in ctx_lens]
    cache = torch.full((sum(pages) + 2, page, 1, D), float("nan"), dtype=torch.bfloat16)
    tables = torch.full((seqs, max(pages)), -1, dtype=torch.int32)
    order = torch.randperm(sum(pages) + 2, generator=g).tolist()
    rows = []
    for s, c in enumerate(ctx_lens):
        keys = torch.randn(c, D, generator=g).to(torch.bfloat16)
        keys[c // 2 :] *= sharp  # later keys stand out
        rows.append(keys.double())
        for b in range(pages[s]):
            tables[s, b] = order.pop()
            part = keys[b * page : (b + 1) * page]
            cache[tables[s, b], : len(part), 0] = part
    qa = (torch.randn(n, heads * D, generator=g) * sharp).to(torch.bfloat16)
    logit = torch.randn(heads, generator=g) if sink else None
    ctx, view = Holder(), Holder()
    ctx.num_seqs, ctx.max_q_len, ctx.max_ctx_len, ctx.status = seqs, max(new), max(ctx_lens), ops.new_status(DEV)
    ctx.tok_seq = torch.cat([torch.full((q,), s, dtype=torch.int32) for s, q in enumerate(new)] + [torch.full((3,), -1, dtype=torch.int32)]).to(DEV)
    ctx.positions = torch.cat([torch.arange(b, b + q, dtype=torch.int32) for b, q in zip(behind, new)] + [torch.zeros(3, dtype=torch.int32)]).to(DEV)
    ctx.q_start = torch.tensor([0] + new).cumsum(0).to(torch.int32).to(DEV)
    view.k_cache, view.block_tables = cache.to(DEV), tables.to(DEV)
    monkeypatch.setattr(latent_ops, "plan_parts", lambda *_: (False, 1))  # (few rows: the keys would be cut for the other kernel)
    got = latent_ops.latent_attention(qa.to(DEV), view, ctx, None if logit is None else logit.to(DEV), heads, rank, rot, scale).double().cpu()
    ops.raise_on_status(ctx.status)
    assert (got[-3:] == 0).all()
    at = 0
    for s, (b, q) in enumerate(zip(behind, new)):
        x = qa[at : at + q].double().view(q, heads, D)
        scores = torch.einsum("qhd,kd->hqk", x, rows[s]) * scale
        hidden = torch.arange(b + q)[None, :] > torch.arange(b, b + q)[:, None]
        scores = scores.masked_fill(hidden, float("-inf"))
        if sink:
            scores = torch.cat([scores, logit.double()[:, None, None].expand(heads, q, 1)], -1)
        weights = torch.softmax(scores, -1)[..., : b + q]
        want = torch.einsum("hqk,kd->qhd", weights, rows[s][:, :rank])
        size = torch.einsum("hqk,kd->qhd", weights, rows[s][:, :rank].abs())
        mine = got[at : at + q].view(q, heads, rank)
        # (a score's own error, D sums of products in float32 against its magnitude, moves its weight by as much)
        slack = D * 2.0**-24 * float(torch.einsum("qhd,kd->hqk", x.abs(), rows[s].abs()).max()) * scale + 2.0**-15
        assert ((mine - want).abs() <= 2.0**-8 * want.abs() + 2 * slack * size + 1e-6).all(), (s, ((mine - want).abs() / (size + 1e-9)).max())
        at += q


def test_a_page_outside_the_pool_is_reported(monkeypatch):
    heads, rank, rot, page = 2, 64, 0, 16
    ctx, view = Holder(), Holder()
    ctx.num_seqs, ctx.max_q_len, ctx.max_ctx_len, ctx.status = 1, 40, 40, ops.new_status(DEV)
    ctx.tok_seq, ctx.positions = torch.zeros(40, dtype=torch.int32, device=DEV), torch.arange(40, dtype=torch.int32, device=DEV)
    ctx.q_start = torch.tensor([0, 40], dtype=torch.int32, device=DEV)
    view.k_cache = torch.zeros(4, page, 1, rank, dtype=torch.bfloat16, device=DEV)
    view.block_tables = torch.tensor([[0, 77, 2]], dtype=torch.int32, device=DEV)
    monkeypatch.setattr(latent_ops, "plan_parts", lambda *_: (False, 1))
    latent_ops.latent_attention(torch.zeros(40, heads * rank, dtype=torch.bfloat16, device=DEV), view, ctx, None, heads, rank, rot, 0.1)
    with pytest.raises(RuntimeError, match="page id outside the pool"):
        ops.raise_on_status(ctx.status)
