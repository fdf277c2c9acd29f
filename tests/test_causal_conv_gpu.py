"""The causal convolution in both its forms (four channels a thread; a channel at a time for other tap counts, widths and alignments)
against float64: portions shorter and longer than the taps, rows kept from before, padding, column slices.  Bound: a chain of
taps + 1 float32 roundings on the sum's terms, silu's own error of a few units in the last place."""

import pytest
import torch

from clockwork_b200.ops import recurrence
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu


class Holder:
    pass


@pytest.mark.parametrize("C, taps, left, extra, offset", [(4, 4, 0, 0, 0), (1028, 4, 4, 8, 12), (4352, 4, 0, 64, 0), (1028, 4, 1, 8, 0), (1028, 4, 0, 8, 2), (30, 4, 0, 2, 0), (512, 3, 0, 0, 0)])
@pytest.mark.parametrize("bias", [False, True])
def test_causal_conv(monkeypatch, C, taps, left, extra, offset, bias):
    g = torch.Generator().manual_seed(C + taps + left)
    new, R = [1, 2, 3, 5, 40], taps - 1
    n = sum(new) + 2
    wide = torch.randn(n, left + C + extra, generator=g)
    weight, b = torch.randn(C, taps, generator=g), torch.randn(C, generator=g) if bias else None
    state = torch.randn(7, offset + R * C + (-(offset + R * C)) % 4, generator=g)
    slots = torch.tensor([3, 0, 6, 2, 5])
    ctx = Holder()
    ctx.tok_seq = torch.cat([torch.full((m,), s, dtype=torch.int32) for s, m in enumerate(new)] + [torch.full((2,), -1, dtype=torch.int32)]).to(DEV)
    ctx.q_start = torch.tensor([0] + new).cumsum(0).to(torch.int32).to(DEV)
    on_device, slots_d = state.to(DEV), slots.to(DEV)
    monkeypatch.setattr(recurrence, "_state_args", lambda _: (on_device.data_ptr(), on_device.stride(0), slots_d.data_ptr()))
    got = recurrence.causal_conv(wide.to(DEV)[:, left : left + C], weight.to(DEV), None if b is None else b.to(DEV), None, offset, ctx).double().cpu()
    assert (got[-2:] == 0).all()
    x, at = wide[:, left : left + C].double(), 0
    for s, m in enumerate(new):
        rows = torch.cat([state[slots[s], offset : offset + R * C].double().view(R, C), x[at : at + m]])
        terms = torch.stack([rows[j : j + m] * weight[:, j].double() for j in range(taps)])
        total, size = terms.sum(0), terms.abs().sum(0)
        if b is not None:
            total, size = total + b.double(), size + b.double().abs()
        want = torch.nn.functional.silu(total)
        # (silu's slope is at most 1.1)
        assert ((got[at : at + m] - want).abs() <= 1.1 * (taps + 1) * 2.0**-24 * size + 2.0**-21 * want.abs() + 1e-30).all(), s
        at += m
