"""Windowed attention on tcgen05 against the same attention in float64: windows of one position, shorter and longer than a tile of
keys and than the contexts, kept first positions in the window's tile and before it, blocks of positions, pages shorter and
longer than a tile, values that are their keys, one to sixteen query heads per key/value head, sizes that fill part of a block of 64
columns, and each switch on the scores and the output.  Keys are not cut, and the kernel is asked
for whatever the step.  Pages that no token
sees are gone from the tables and the cache holds NaN wherever no token was stored.  Bound: sums of bfloat16 operands in float32,
weights in two bfloat16 halves (2^-16), the result rounded to bfloat16 (2^-8)."""

import pytest
import torch

from clockwork_b200 import ops
from clockwork_b200.ops import window as window_ops
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, G, dk, dv, voff, window, keep, blocked, page, extras", [
    (16, 4, 128, 128, 128, 100, 4, False, 16, ""),
    (16, 4, 128, 128, 64, 333, 0, False, 32, "sink gate_entry"),
    (8, 8, 64, 48, 64, 1, 0, False, 8, "head_scale"),
    (32, 2, 16, 16, 16, 64, 70, False, 64, "sink head_bias"),
    (16, 4, 48, 80, 48, 130, 0, True, 16, "sink gate temperature"),
    (16, 4, 128, 64, 128, 1 << 30, 0, False, 128, "head_scale gate"),
])
def test_portions(H, G, dk, dv, voff, window, keep, blocked, page, extras):
    g = torch.Generator().manual_seed(H + dk + window % 1000)
    per, width = H // G, voff + dv
    behind, new = [0, 37, 500, 3], [300, 129, 260, 1]
    new.append(max(1, 64 * 128 // H - sum(new) + 40))
    behind.append(0)
    n = sum(new) + 3
    ctx_lens = [b + q for b, q in zip(behind, new)]
    pages = [-(-c // page) for c in ctx_lens]
    cache = torch.full((sum(pages) + 2, page, G, width), float("nan"), dtype=torch.bfloat16)
    tables = torch.full((len(new), max(pages)), -1, dtype=torch.int32)
    order = torch.randperm(sum(pages) + 2, generator=g).tolist()
    rows = []
    for s, c in enumerate(ctx_lens):
        row = torch.randn(c, G, width, generator=g).to(torch.bfloat16)
        row[c // 2 :] *= 2  # later keys stand out
        rows.append(row.double())
        first = behind[s] - behind[s] % window if blocked else max(0, behind[s] - window + 1)
        for b in range(pages[s]):
            if (b + 1) * page <= first and b * page >= keep:
                continue  # given back
            tables[s, b] = order.pop()
            part = row[b * page : (b + 1) * page]
            cache[tables[s, b], : len(part)] = part
    q = torch.randn(n, H * dk + 8, generator=g).to(torch.bfloat16)
    tok_seq = torch.cat([torch.full((m,), s, dtype=torch.int32) for s, m in enumerate(new)] + [torch.full((3,), -1, dtype=torch.int32)]).to(DEV)
    positions = torch.cat([torch.arange(b, b + m, dtype=torch.int32) for b, m in zip(behind, new)] + [torch.zeros(3, dtype=torch.int32)]).to(DEV)
    q_start = torch.tensor([0] + new).cumsum(0).to(torch.int32).to(DEV)
    draw = lambda *size: torch.randn(*size, generator=g)  # noqa: E731
    head_scale = draw(H) if "head_scale" in extras else None  # (negative ones among them)
    if head_scale is not None:
        head_scale[1] = 0.0
    head_bias = draw(H) if "head_bias" in extras else None
    sink = draw(H) if "sink" in extras else None
    temperature = (0.3, 50) if "temperature" in extras else None
    entries = "gate_entry" in extras
    gate = draw(n, H * dv if entries else H) if "gate" in extras else None
    scale = dk**-0.5
    on = lambda t: None if t is None else t.to(DEV)  # noqa: E731
    status = ops.new_status(DEV)
    window_ops.set_tensor_cores(3)  # (this kernel, where another would be faster as well)
    try:
        got = window_ops.window_attention(q.to(DEV), cache.to(DEV), tables.to(DEV), positions, tok_seq, q_start, H, G, dk, dv, window, scale,
                                          on(head_scale), None, on(head_bias), False, status, 1, blocked=blocked, sink=on(sink),
                                          temperature=temperature, gate=on(gate), keep_first=keep, value_offset=voff,
                                          gate_entries=entries).double().cpu()
    finally:
        window_ops.set_tensor_cores(True)
    ops.raise_on_status(status)
    assert (got[-3:] == 0).all()
    at = 0
    for s, (b, m) in enumerate(zip(behind, new)):
        x = q[at : at + m, : H * dk].double().view(m, H, dk)
        k, v = (rows[s][:, :, i : i + d].repeat_interleave(per, 1) for i, d in ((0, dk), (voff, dv)))
        t, j = torch.arange(b, b + m)[:, None], torch.arange(b + m)[None, :]
        seen = (j <= t) & ((j >= t - t % window) if blocked else ((t - j < window) | (j < keep)))
        factor = torch.full((H, m, 1), scale, dtype=torch.float64)
        if head_scale is not None:
            factor = factor * head_scale.double()[:, None, None]
        if temperature:
            factor = factor * (1 + temperature[0] * torch.log(torch.floor((t.double() + 1) / temperature[1]) + 1))
        scores = torch.einsum("qhd,khd->hqk", x, k) * factor
        if head_bias is not None:
            scores = scores + head_bias.double()[:, None, None]
        size = torch.einsum("qhd,khd->hqk", x.abs(), k.abs()).max() * float(factor.abs().max())
        scores = scores.masked_fill(~seen, float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink.double()[:, None, None].expand(H, m, 1)], -1)
        weights = torch.softmax(scores, -1)[..., : b + m]
        want, total = (torch.einsum("hqk,khd->qhd", weights, z) for z in (v, v.abs()))
        if gate is not None:
            open_ = torch.sigmoid(gate[at : at + m].double()).view(m, H, dv if entries else 1)
            want, total = want * open_, total * open_
        mine = got[at : at + m].view(m, H, dv)
        # (a score's own error, dk sums of products in float32 and the factor's rounding, moves its weight by as much)
        slack = (dk + 4) * 2.0**-24 * float(size) + 2.0**-15
        off = (mine - want).abs()
        assert (off <= 2.0**-8 * want.abs() + 2 * slack * total + 1e-6).all(), (s, float((off / (total + 1e-9)).max()))
        at += m


@pytest.mark.parametrize("H, G, d, window, behind, new, here", [
    # uncut: windows and counts of single tokens on both sides of the rule
    (16, 4, 128, 64, 1500, [1] * 64, False), (16, 4, 128, 128, 1500, [1] * 64, True), (16, 4, 128, 128, 1500, [1] * 128, False),
    (32, 8, 64, 256, 1500, [1] * 128, False), (32, 8, 64, 320, 1500, [1] * 128, True), (16, 16, 64, 64, 1500, [1] * 8, True),
    (8, 8, 128, 64, 1500, [1] * 48, False), (64, 8, 64, 128, 1500, [1] * 64, True),
    # portions in narrow windows
    (16, 4, 128, 32, 0, [300], False), (16, 4, 128, 64, 0, [300], True), (16, 4, 64, 64, 500, [40], False),
    # cut in up to four parts, and in more on few and on many row tiles
    (32, 8, 64, 512, 1500, [1] * 8, False), (32, 8, 64, 512, 1500, [1] * 24, True), (32, 8, 64, 512, 1500, [32], False),
    (16, 4, 128, 512, 1500, [1] * 8, True), (16, 4, 128, 1024, 1500, [1] * 8, False), (16, 4, 128, 1 << 30, 8000, [64], False),
    (16, 4, 128, 1 << 30, 8000, [512], True),
    # query heads that the mma.sync kernel does not take
    (32, 1, 64, 64, 500, [1] * 4, True),
])
def test_the_rule_between_the_kernels(H, G, d, window, behind, new, here):
    """Steps on both sides of every line of the rule that chooses between the two tensor-core kernels: the default gives the bits of
    the kernel that the rule names, and the two agree (weights in two bfloat16 halves and sums in float32 in both, the results rounded
    to bfloat16: 2^-8 of the value from each, and 2^-15 of the sum of magnitudes)."""
    page, n = 16, sum(new)
    pages = -(-(behind + max(new)) // page)
    g = torch.Generator(device=DEV).manual_seed(window % 997 + n)
    cache = torch.randn(pages, page, G, 2 * d, device=DEV, generator=g).bfloat16()  # (the requests share their pages)
    tables = torch.arange(pages, dtype=torch.int32, device=DEV).expand(len(new), pages).contiguous()
    tok_seq = torch.repeat_interleave(torch.arange(len(new), dtype=torch.int32), torch.tensor(new)).to(DEV)
    positions = torch.cat([torch.arange(behind, behind + m, dtype=torch.int32) for m in new]).to(DEV)
    q_start = torch.tensor([0] + new).cumsum(0).to(torch.int32).to(DEV)
    q, status = torch.randn(n, H * d, device=DEV, generator=g).bfloat16(), ops.new_status(DEV)
    parts = window_ops.window_parts(n, window, torch.bfloat16, behind + max(new))
    outs = {}
    try:
        for mode in (1, 2, 3):
            window_ops.set_tensor_cores(mode)
            outs[mode] = window_ops.window_attention(q, cache, tables, positions, tok_seq, q_start, H, G, d, d, window, d**-0.5, None, None, None,
                                                     False, status, parts)
    finally:
        window_ops.set_tensor_cores(True)
    ops.raise_on_status(status)
    assert torch.equal(outs[1], outs[3 if here else 2])
    assert not torch.equal(outs[2], outs[3]) or window == 1
    size = float(cache.float().abs().mean()) + 1
    off = (outs[2].double() - outs[3].double()).abs()
    assert (off <= 2 * 2.0**-8 * outs[3].double().abs() + 2.0**-13 * size).all(), float(off.max())
