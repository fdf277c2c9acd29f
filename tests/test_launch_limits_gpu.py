"""Launches of different sizes of one kernel from two host threads, each on a stream of its own.  A launcher that set the kernel's limit
of dynamic shared memory to what its own call needs could lower it between the other thread's setting and its launch, which then fails."""

import threading

import pytest
import torch

from clockwork_b200 import ops
from clockwork_b200.ops import grouped, latent, recurrence, window
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu
PAGE, PAGES = 16, 20


class Holder:
    pass


def one_request(n):
    ctx, view = Holder(), Holder()
    ctx.num_seqs, ctx.max_q_len, ctx.max_ctx_len, ctx.status = 1, n, n, ops.new_status(DEV)
    ctx.tok_seq, ctx.positions = torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    ctx.q_start = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    view.block_tables = torch.arange(PAGES, dtype=torch.int32, device=DEV)[None]
    return ctx, view


def chunk_scan(n):
    ctx, view = one_request(n)
    view.state, view.slots, view.slots_host = torch.zeros(1, 2 * 128 * 16, device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV), []
    qk, v = torch.randn(n, 512, device=DEV), torch.randn(n, 32, device=DEV)
    return lambda: recurrence.recurrence_scan(recurrence.FORM_HEAD_DECAY, qk[:, :256], qk[:, 256:], v, None, torch.full((2,), 0.9, device=DEV), None,
                                              None, view, 0, ctx, 2, 128, 16, chunks=True)


def float32_rows(hd):
    ctx, view = one_request(100)
    q, cache = torch.randn(100, 2 * hd, device=DEV), torch.randn(PAGES, PAGE, 1, hd, device=DEV)
    return lambda: ops.attention_ref(q, cache, cache, view.block_tables, ctx.tok_seq, ctx.positions, 2, 1, hd, 0.1, None, ctx.status,
                                     ctx.q_start)


def windowed(d):
    ctx, view = one_request(100)
    q, cache = torch.randn(100, 2 * d, device=DEV).bfloat16(), torch.randn(PAGES, PAGE, 1, 2 * d, device=DEV).bfloat16()
    return lambda: window.window_attention(q, cache, view.block_tables, ctx.positions, ctx.tok_seq, ctx.q_start, 2, 1, d, d, 1000, 0.1, None, None,
                                           None, False, ctx.status, 1)


def over_a_latent(rank):
    ctx, view = one_request(100)
    ctx.max_ctx_len = 64  # (uncut keys)
    view.k_cache = torch.randn(PAGES, PAGE, 1, rank + 64, device=DEV).bfloat16()
    qa = torch.randn(100, 2 * (rank + 64), device=DEV).bfloat16()
    return lambda: latent.latent_attention(qa, view, ctx, None, 2, rank, 64, 0.1)


def in_groups(groups):
    rows = torch.randn(groups, 64, device=DEV).bfloat16()
    w = torch.randn(groups, 64, 64, device=DEV).bfloat16()
    at = torch.arange(groups + 1, dtype=torch.int32, device=DEV)
    return lambda: grouped.expert_down(rows, w, at, at[:groups])


KERNELS = [
    (recurrence, "cw_chunk_scan", chunk_scan, 300, 40),
    (ops, "cw_attention_rows", float32_rows, 128, 64),
    (window, "cw_window_attention", windowed, 128, 64),
    (latent, "cw_latent_attention", over_a_latent, 512, 64),
    (grouped, "cw_grouped_gemm", in_groups, 1024, 4),
]


def recorded(monkeypatch, module, name, make, sizes):
    """The library's calls for these sizes, each on a stream of its own, with their arguments; and every buffer that they point at."""
    real, empty = module.library(), torch.empty
    calls, kept = [], []

    class Recorder:
        def __getattr__(self, function):
            def call(*args):
                if function == name:
                    calls.append((getattr(real, function), args))
                return getattr(real, function)(*args)
            return call

    def keep(*args, **kwargs):
        kept.append(empty(*args, **kwargs))
        return kept[-1]

    monkeypatch.setattr(module, "library", Recorder)
    monkeypatch.setattr(torch, "empty", keep)
    for size in sizes:
        with torch.cuda.stream(torch.cuda.Stream()):
            step = make(size)
            kept += [step, step()]
    torch.cuda.synchronize()
    monkeypatch.undo()
    assert len(calls) == len(sizes)
    return calls, kept


@pytest.mark.parametrize("module, name, make, large, small", KERNELS, ids=[k[1] for k in KERNELS])
def test_two_threads(monkeypatch, module, name, make, large, small):
    calls, kept = recorded(monkeypatch, module, name, make, (large, small))
    before = [t.clone() for t in kept if isinstance(t, torch.Tensor)]
    refused = []

    def replay(function, args):
        torch.cuda.set_device(0)
        for _ in range(4000):
            rc = function(*args)
            if rc:
                refused.append(rc)

    threads = [threading.Thread(target=replay, args=call) for call in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not refused, (len(refused), refused[0])
    if name != "cw_chunk_scan":  # (whose state moves on with every call)
        assert all(torch.equal(a, b) for a, b in zip(before, (t for t in kept if isinstance(t, torch.Tensor))))


@pytest.mark.parametrize("module, name, make, large, small", KERNELS, ids=[k[1] for k in KERNELS])
def test_a_thread_that_has_not_used_the_gpu(monkeypatch, module, name, make, large, small):
    """(The tensor maps' encoder wants the device's context in the calling thread, which a launch would have put there.)"""
    calls, kept = recorded(monkeypatch, module, name, make, (large,))
    answers = []
    thread = threading.Thread(target=lambda: answers.append(calls[0][0](*calls[0][1])))
    thread.start()
    thread.join()
    torch.cuda.synchronize()
    assert answers == [0] and kept
