"""The tcgen05 products in groups at the edges of their tiles, against the same sums in float64: groups without rows, of one row,
around multiples of 16 (a tile's width), of 32, 128 and 256 (the widest tiles); feature counts and inner sizes that end within a
tile; every epilogue.  Bound: operands are bfloat16, sums float32 (2^-24 per term of the sum of magnitudes), results rounded to
bfloat16 (2^-8 of the value, a unit of the gate's own rounding with it) or kept in float32."""

import pytest
import torch

from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu
FEW = [0, 1, 15, 16, 17, 0, 31, 32, 33, 64]          # 21 rows a group on average: the narrow tiles
MANY = [127, 0, 128, 129, 1, 255, 256, 257, 300, 16]  # 147 on average: the wide ones


def close(got, want, magnitude, k):
    bound = (k * 2.0**-24) * magnitude + (2.0**-8 * want.abs() if got.dtype == torch.bfloat16 else 0) + 1e-30
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() / bound).max()


def operands(sizes, top, n, k, seed=0):
    g = torch.Generator().manual_seed(seed)
    experts, pairs = len(sizes), sum(sizes)
    tokens = -(-pairs // top)
    x = torch.randn(tokens, k, generator=g).to(torch.bfloat16).to(DEV)
    offsets = torch.tensor([0] + sizes).cumsum(0).to(torch.int32).to(DEV)
    order = torch.randperm(pairs, generator=g).to(torch.int32).to(DEV)
    w = [(torch.randn(experts, n, k, generator=g) * k**-0.5).to(torch.bfloat16).to(DEV) for _ in range(2)]
    group = torch.repeat_interleave(torch.arange(experts), torch.tensor(sizes)).to(DEV)
    return x, offsets, order, w, group


def per_group(rows, w, group):
    """float64 products of row r with the matrix of its group, and the sums of magnitudes."""
    want = torch.empty(rows.shape[0], w.shape[1], dtype=torch.float64, device=DEV)
    size = torch.empty_like(want)
    for g in range(w.shape[0]):
        at = group == g
        want[at] = rows[at].double() @ w[g].double().T
        size[at] = rows[at].double().abs() @ w[g].double().abs().T
    return want, size


def gate_and_up(x, wg, wu, offsets, order, top, a, a_size, b, b_size, k):
    """The two products that begin an expert, given their sums in float64 (a: gate, b: up) and the sums of magnitudes."""
    from clockwork_b200.ops import grouped

    silu = torch.nn.functional.silu
    # |silu'| <= 1.1, |silu(a)| <= |a|: what the two sums' errors become in the product
    close(grouped.expert_gate_up(x, wg, wu, offsets, order, top), silu(a) * b, 1.1 * a_size * b.abs() + silu(a).abs() * b_size + 1e-6 * (a * b).abs(), 2 * k)
    close(grouped.expert_up_relu2(x, wu, offsets, order, top), b.clamp(min=0) ** 2, 2 * b.clamp(min=0) * b_size, 2 * k)


@pytest.mark.parametrize("sizes", [FEW, MANY], ids=["few", "many"])
@pytest.mark.parametrize("n,k", [(200, 72), (256, 640)])
def test_experts(sizes, n, k):
    from clockwork_b200.ops import grouped

    top = 3
    x, offsets, order, (wg, wu), group = operands(sizes, top, n, k)
    rows = x[order.long() // top]
    (a, a_size), (b, b_size) = per_group(rows, wg, group), per_group(rows, wu, group)
    gate_and_up(x, wg, wu, offsets, order, top, a, a_size, b, b_size, k)
    act = torch.randn(sum(sizes), k, device=DEV).to(torch.bfloat16)
    y, y_size = per_group(act, wu, group)
    want, size = torch.empty_like(y), torch.empty_like(y)
    want[order.long()], size[order.long()] = y, y_size  # rows are written in pair order
    close(grouped.expert_down(act, wu, offsets, order), want, size, k)


@pytest.mark.parametrize("rows", [1, 32, 33, 257])
@pytest.mark.parametrize("gate", ["none", "entry", "head"])
def test_per_head(rows, gate):
    from clockwork_b200.ops import grouped

    heads, n, k, a_width, out_width = 5, 130, 128, 192, 136
    g = torch.Generator().manual_seed(rows)
    a = torch.randn(rows, heads * a_width, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(heads, n, k, generator=g) * k**-0.5).to(torch.bfloat16).to(DEV)
    out = torch.full((rows, heads * out_width), 7.0, dtype=torch.bfloat16, device=DEV)
    kwargs, factor = {}, torch.ones(rows, heads, n, dtype=torch.float64, device=DEV)
    if gate == "entry":
        kwargs["gate"] = torch.randn(rows, heads * out_width, generator=g).to(torch.bfloat16).to(DEV)
        factor = torch.sigmoid(kwargs["gate"].double().view(rows, heads, out_width)[..., :n])
    if gate == "head":
        kwargs["head_gate"] = torch.randn(rows, heads + 2, generator=g).to(DEV)
        factor = torch.sigmoid(kwargs["head_gate"].double()[:, :heads, None])
    grouped.per_head_product(a, a_width, w, out, out_width, **kwargs)
    rows_of = a.double().view(rows, heads, a_width)[..., :k]
    want = torch.einsum("rhk,hnk->rhn", rows_of, w.double())
    size = torch.einsum("rhk,hnk->rhn", rows_of.abs(), w.double().abs())
    got = out.view(rows, heads, out_width)
    close(got[..., :n], want * factor, (size + 8 * want.abs()) * factor, k)
    assert (got[..., n:] == 7.0).all()  # nothing beyond a head's own columns


def test_takes_and_leaves():
    """The forms that TMA cannot address go to the other kernels and agree with the ones it can: an inner size that is no
    multiple of 8, a row base off a 16-byte boundary, an odd number of features."""
    from clockwork_b200.ops import grouped

    for n, k in ((129, 64), (64, 36), (64, 64)):
        x, offsets, order, (wg, _), group = operands(MANY, 1, n, k, seed=n + k)
        base = torch.zeros(wg.numel() + 1, dtype=torch.bfloat16, device=DEV)
        shifted = base[1:].view(wg.shape).copy_(wg) if (n, k) == (64, 64) else wg
        want, size = per_group(x[order.long()], wg, group)
        act = x[order.long()].contiguous()
        close(grouped.expert_down(act, shifted, offsets, torch.arange(sum(MANY), dtype=torch.int32, device=DEV)), want, size, k)
        gate_and_up(x, shifted, shifted, offsets, order, 1, want, size, want, size, k)
