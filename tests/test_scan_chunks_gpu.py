"""Recurrences with one decay per head, a portion's tokens 16 at a time, against the same recurrence in float64 and beside the form
that takes them one by one: portions of one token, at the edges of a chunk and of many chunks, requests without tokens, padding
rows, columns that end within a block, heads that share keys, states that are not zero, decays near one and near zero.  Bound: both
forms add the same float32 terms in another order, so the chunks may be twice as far from float64 as the other form is at its
worst, and no closer bound than 2^-20 of the largest value is asked."""

import pytest
import torch

from clockwork_b200.ops import recurrence as rec
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu
LENS, PAD, TAPS = [1, 15, 0, 16, 17, 130, 33], 3, 4
N = sum(LENS) + PAD


class View:
    def __init__(self, state):
        self.state, self.slots, self.slots_host = state, torch.arange(len(LENS), device=DEV), []


class Context:
    num_seqs = len(LENS)

    def __init__(self):
        self.tok_seq = torch.cat([torch.full((m,), s, dtype=torch.int32) for s, m in enumerate(LENS)]
                                 + [torch.full((PAD,), -1, dtype=torch.int32)]).to(DEV)
        self.q_start = torch.tensor([0] + LENS).cumsum(0).to(torch.int32).to(DEV)


def recurrence(q, k, v, a, b, s, delta):
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        s = s * a[t][:, None, None]
        u = b[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", s, k[t]) if delta else v[t])
        s = s + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", s, q[t])
    return out, s


def compare(outs, states, want, last):
    for got, right in ((outs, want), (states, last)):
        off = {c: float((got[c] - right).abs().max()) for c in got}
        assert off[True] <= 2 * off[False] + 2.0**-20 * float(right.abs().max()), off


@pytest.mark.parametrize("groups, heads, dk, dv", [(2, 4, 128, 128), (3, 3, 32, 17), (1, 2, 64, 33), (1, 3, 128, 5)])
def test_delta_rule(groups, heads, dk, dv):
    g = torch.Generator().manual_seed(dk + dv)
    qk = groups * dk
    channels, kept = 2 * qk + heads * dv, heads * dk * dv
    x, conv = torch.randn(N, channels, generator=g), torch.randn(channels, TAPS, generator=g) * 0.5
    beta, decay = torch.randn(N, heads, generator=g), torch.randn(N, heads, generator=g) * 3
    dt_bias, a_log = torch.randn(heads, generator=g) - 2, torch.linspace(-3, 2.5, heads)
    start = torch.randn(len(LENS) + 1, kept + (TAPS - 1) * channels, generator=g) * 0.3
    ctx, outs, states = Context(), {}, {}
    for chunks in (False, True):
        view = View(start.clone().to(DEV))
        outs[chunks] = rec.head_delta(x.to(DEV), conv.to(DEV), beta.to(DEV), decay.to(DEV), dt_bias.to(DEV), a_log.to(DEV), view, 0, kept, ctx,
                                      groups, heads, dk, dv, 1e-6, dk**-0.5, chunks=chunks)[: N - PAD].double().cpu()
        states[chunks] = view.state.double().cpu()
    want, last, at = torch.empty(N - PAD, heads * dv, dtype=torch.float64), start.double().clone(), 0
    for s, m in enumerate(LENS):
        if not m:
            continue
        cv = conv.double()
        before = torch.cat([start[s, kept:].double().view(TAPS - 1, channels), x[at : at + m].double()])
        y = torch.nn.functional.silu(sum(before[j : j + m] * cv[:, j] for j in range(TAPS)))
        q, k, v = y[:, :qk].view(m, groups, dk), y[:, qk : 2 * qk].view(m, groups, dk), y[:, 2 * qk :].view(m, heads, dv)
        q, k = (z / torch.sqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q, k = ((z * f).repeat_interleave(heads // groups, 1) for z, f in ((q, dk**-0.5), (k, 1.0)))
        a = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(decay[at : at + m].double() + dt_bias.double(), threshold=1e9))
        s0 = start[s, :kept].double().view(heads, dv, dk).transpose(1, 2)
        y, s1 = recurrence(q, k, v, a, torch.sigmoid(beta[at : at + m].double()), s0, True)
        want[at : at + m] = y.reshape(m, -1)
        last[s, :kept] = s1.transpose(1, 2).reshape(-1)
        last[s, kept:] = before[-(TAPS - 1) :].reshape(-1)
        at += m
    compare(outs, states, want, last)


@pytest.mark.parametrize("form", ["step size", "constant", "gated"])
@pytest.mark.parametrize("groups, heads, dk, dv", [(1, 4, 128, 64), (3, 3, 32, 17), (2, 2, 64, 33)])
def test_one_decay_per_head(form, groups, heads, dk, dv):
    g = torch.Generator().manual_seed(dk + dv)
    wide = torch.randn(N, 2 * groups * dk + 4, generator=g)  # (q and k lie in a wider matrix)
    v = torch.randn(N, heads * (dv - (form == "gated")), generator=g)
    start = torch.randn(len(LENS) + 1, heads * dk * dv, generator=g) * 0.3
    decays, q_scale, skip = torch.linspace(0.3, 0.9999, heads), 0.7, None
    pre, dt_bias, a_log = torch.randn(N, heads, generator=g), torch.randn(heads, generator=g) - 3, torch.linspace(-2, 2.5, heads)
    if form == "step size":
        q_scale, skip = 1.0, torch.randn(heads, generator=g)
        b = torch.nn.functional.softplus(pre.double() + dt_bias.double(), threshold=1e9)
        a = torch.exp(-torch.exp(a_log.double()) * b)
        args = (rec.FORM_STEP_SIZE, dict(pre=pre, p0=dt_bias, p1=a_log, p2=skip))
    elif form == "constant":
        a, b = decays.double().expand(N, heads), torch.ones(N, heads, dtype=torch.float64)
        args = (rec.FORM_HEAD_DECAY, dict(pre=None, p0=decays, p1=None, p2=None))
    else:
        coef = torch.rand(N, 3 * heads, generator=g)
        a, b = coef[:, :heads].double(), coef[:, heads : 2 * heads].double()
        args = (rec.FORM_GATED_WITH_KEY_SUM, dict(pre=coef, p0=None, p1=None, p2=None))
    on = lambda t: None if t is None else t.to(DEV)  # noqa: E731
    ctx, outs, states = Context(), {}, {}
    for chunks in (False, True):
        view, w = View(start.clone().to(DEV)), wide.to(DEV)
        outs[chunks] = rec.recurrence_scan(args[0], w[:, : groups * dk], w[:, groups * dk : 2 * groups * dk], v.to(DEV), view=view, offset=0, ctx=ctx,
                                           heads=heads, dk=dk, dv=dv, heads_per_group=heads // groups, q_scale=q_scale, chunks=chunks,
                                           **{name: on(t) for name, t in args[1].items()})[: N - PAD].double().cpu()
        states[chunks] = view.state.double().cpu()
    want, last, at = torch.empty(N - PAD, heads * dv, dtype=torch.float64), start.double().clone(), 0
    for s, m in enumerate(LENS):
        if not m:
            continue
        q, k = (wide[at : at + m, i * groups * dk : (i + 1) * groups * dk].double().view(m, groups, dk).repeat_interleave(heads // groups, 1)
                for i in (0, 1))
        vs = v[at : at + m].double().view(m, heads, -1)
        if form == "gated":
            vs = torch.cat([vs, torch.ones(m, heads, 1, dtype=torch.float64)], -1)
        y, s1 = recurrence(q, k, vs, a[at : at + m], b[at : at + m], start[s].double().view(heads, dv, dk).transpose(1, 2), False)
        y = q_scale * y + (0 if skip is None else skip.double()[:, None] * vs)
        want[at : at + m] = y.reshape(m, -1)
        last[s] = s1.transpose(1, 2).reshape(-1)
        at += m
    compare(outs, states, want, last)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("form", ["delta", "step size", "constant", "gated"])
@pytest.mark.parametrize("operand", ["q", "k", "v"])
def test_a_token_that_is_not_finite_does_not_reach_earlier_ones(form, operand, bad):
    """Outputs of the tokens before it, of a chunk that it shares with them and of the chunks before, keep their bits; so do the
    other requests' outputs and states."""
    groups, heads, dk, dv = 2, 2, 64, 32
    g = torch.Generator().manual_seed(5)
    qk, ones = groups * dk, form == "gated"
    start_of, spoiled = sum(LENS[:5]), 5  # the request of 130 tokens; its 40th token, in the middle of a chunk
    at = start_of + 39
    x = torch.randn(N, 2 * qk + heads * (dv - ones), generator=g)
    conv = torch.zeros(x.shape[1], TAPS)
    conv[:, -1] = 1.0  # (the delta layer's convolution passes its current input on alone)
    coef, decays = torch.rand(N, 3 * heads, generator=g), torch.linspace(0.5, 0.99, heads)
    state = torch.randn(len(LENS) + 1, heads * dk * dv + (TAPS - 1) * x.shape[1], generator=g) * 0.3
    on = lambda t: None if t is None else t.clone().to(DEV)  # noqa: E731
    ctx, outs, states = Context(), [], []
    for value in (None, bad):
        rows, view = x.clone(), View(on(state))
        if value is not None:
            rows[at, {"q": 3, "k": qk + 3, "v": 2 * qk + 3}[operand]] = value
        w = on(rows)
        if form == "delta":
            out = rec.head_delta(w, on(conv), on(coef[:, :heads]), on(coef[:, heads : 2 * heads]), on(decays - 2), on(decays - 1), view, 0, heads * dk * dv, ctx,
                                 groups, heads, dk, dv, 1e-6, 1.0, chunks=True)
        else:
            number, args = {"step size": (rec.FORM_STEP_SIZE, dict(pre=coef[:, :heads].contiguous(), p0=decays, p1=decays, p2=decays)),
                            "constant": (rec.FORM_HEAD_DECAY, dict(pre=None, p0=decays, p1=None, p2=None)),
                            "gated": (rec.FORM_GATED_WITH_KEY_SUM, dict(pre=coef, p0=None, p1=None, p2=None))}[form]
            out = rec.recurrence_scan(number, w[:, :qk], w[:, qk : 2 * qk], w[:, 2 * qk :], view=view, offset=0, ctx=ctx, heads=heads, dk=dk, dv=dv,
                                      heads_per_group=heads // groups, chunks=True, **{name: on(t) for name, t in args.items()})
        outs.append(out.cpu())
        states.append(view.state.cpu())
    end = start_of + LENS[spoiled]
    assert torch.isfinite(outs[0][: N - PAD]).all()
    assert torch.equal(outs[1][:at], outs[0][:at]) and torch.equal(outs[1][end : N - PAD], outs[0][end : N - PAD])
    assert not torch.isfinite(outs[1][at:end]).all()  # (it does reach its own output or later ones)
    others = [s for s in range(len(LENS)) if s != spoiled]
    assert torch.equal(states[1][others], states[0][others])


@pytest.mark.parametrize("form", ["delta", "step size", "constant", "gated"])
def test_single_tokens_beside_portions_keep_their_bits(form):
    """With chunks from two tokens on, a request of one token gets the bits of the scan that takes tokens one by one, as in a step
    of single tokens, and every other request those of the chunks; nobody's state is moved on twice."""
    groups, heads, dk, dv = 2, 4, 64, 48
    g = torch.Generator().manual_seed(6)
    qk, ones = groups * dk, form == "gated"
    x = torch.randn(N, 2 * qk + heads * (dv - ones), generator=g)
    conv, coef = torch.randn(x.shape[1], TAPS, generator=g) * 0.5, torch.rand(N, 3 * heads, generator=g)
    decays = torch.linspace(0.5, 0.99, heads)
    state = torch.randn(len(LENS) + 1, heads * dk * dv + (TAPS - 1) * x.shape[1], generator=g) * 0.3
    on = lambda t: None if t is None else t.clone().to(DEV)  # noqa: E731
    ctx, outs, states = Context(), {}, {}
    for chunks in (0, 1, 2):
        w, view = on(x), View(on(state))
        if form == "delta":
            out = rec.head_delta(w, on(conv), on(coef[:, :heads]), on(coef[:, heads : 2 * heads]), on(decays - 2), on(decays - 1), view, 0,
                                 heads * dk * dv, ctx, groups, heads, dk, dv, 1e-6, 1.0, chunks=chunks)
        else:
            number, args = {"step size": (rec.FORM_STEP_SIZE, dict(pre=coef[:, :heads].contiguous(), p0=decays, p1=decays, p2=decays)),
                            "constant": (rec.FORM_HEAD_DECAY, dict(pre=None, p0=decays, p1=None, p2=None)),
                            "gated": (rec.FORM_GATED_WITH_KEY_SUM, dict(pre=coef, p0=None, p1=None, p2=None))}[form]
            out = rec.recurrence_scan(number, w[:, :qk], w[:, qk : 2 * qk], w[:, 2 * qk :], view=view, offset=0, ctx=ctx, heads=heads, dk=dk, dv=dv,
                                      heads_per_group=heads // groups, chunks=chunks, **{name: on(t) for name, t in args.items()})
        outs[chunks], states[chunks] = out.cpu(), view.state.cpu()
    at = 0
    for s, m in enumerate(LENS):
        right = 0 if m == 1 else 1
        assert torch.equal(outs[2][at : at + m], outs[right][at : at + m]) and torch.equal(states[2][s], states[right][s]), (s, m)
        at += m
    assert not torch.equal(outs[0], outs[1])
