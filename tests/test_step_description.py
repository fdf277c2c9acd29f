"""The host's description of a step that replays a captured graph, against the same arrays written number by number, over one and many
requests, portions and single tokens, places wanted of none, one and all, page groups of one row per position and per several.
The host work is part of the time to a prompt's first token: it may not take longer than the plain lines do."""

import time
from types import MethodType, SimpleNamespace

import numpy as np
import pytest

from clockwork_b200.cache import NO_PAGE
from clockwork_b200.engine import step
from clockwork_b200.engine.step import PortionGraph, StepEntry

PAGE, EVERY, SCRATCH = 16, (1, 6), 63
LAYOUTS = {"one prompt": ([32], [0]), "one long prompt": ([2048], [0]), "behind a context": ([2003], [777]),
           "ragged prompts": ([900, 333, 65], [0, 15, 16]), "mixed": ([391, 1, 130, 1, 1, 2], [0, 500, 517, 31, 32, 95]),
           "many single tokens": ([40] + [1] * 50, [7] + [1000 + 3 * i for i in range(50)])}


def make(layout, want):
    new, behind = LAYOUTS[layout]
    entries, reqs, at = [], [], 0
    for i, (n, b) in enumerate(zip(new, behind)):
        places = {"none": [], "last": [n - 1], "all": list(range(n)), "some": [0, n - 1, n // 2] if i % 2 else []}[want]
        entries.append(StepEntry(str(i), [(37 * j + 11 * i) % 151000 for j in range(n)], places))
        tables = []
        for every in EVERY:
            pages = -(-(b + n + 40) // every // PAGE) + 1  # (some reserved ahead)
            tables.append([at + (7 * k) % pages for k in range(pages)])
            tables[-1][: b // every // PAGE] = [NO_PAGE] * (b // every // PAGE)  # given back
            at += pages
        reqs.append(SimpleNamespace(request_id=str(i), num_computed=b, tables=tables, state_slot=None if i % 3 == 2 else i))
    cache = SimpleNamespace(page_size=PAGE, groups=[SimpleNamespace(every=e) for e in EVERY], state=SimpleNamespace(scratch_slot=SCRATCH))
    tokens, seqs = sum(new) + 13, len(new) + 2
    graph = SimpleNamespace(_uploaded=SimpleNamespace(synchronize=lambda: None), _scalar_rules={}, _arrays={}, max_blocks=200)
    sizes = dict(tokens=tokens, positions=tokens, tok_seq=tokens, q_start=seqs + 1, ctx_lens=seqs, rows=tokens, state=seqs)
    graph.h = {name: np.full(n, 12345, np.int32) for name, n in sizes.items()}
    for g in range(len(EVERY)):
        graph.h[f"slots{g}"], graph.h[f"tables{g}"] = np.full(tokens, 12345, np.int32), np.full((seqs, graph.max_blocks), 12345, np.int32)
    graph._write_padding = MethodType(PortionGraph._write_padding, graph)
    return graph, cache, entries, reqs


def describe(graph, cache, entries, reqs):
    firsts = step._firsts(entries)
    return PortionGraph.fill(graph, cache, entries, reqs, firsts, step._wanted_rows(entries, firsts))


def plain(graph, cache, entries, reqs):
    h, at, wanted = graph.h, 0, 0
    q_start = np.zeros(len(entries) + 1, np.int32)
    q_start[1:] = np.cumsum([len(e.tokens) for e in entries])
    h["tokens"][: q_start[-1]] = np.fromiter((t for e in entries for t in e.tokens), dtype=np.int64, count=q_start[-1])
    h["q_start"][: len(q_start)] = q_start
    rows = [int(q_start[i]) + w for i, e in enumerate(entries) for w in e.want]
    h["rows"][: len(rows)] = rows
    for i, (e, r) in enumerate(zip(entries, reqs)):
        at, end = int(q_start[i]), int(q_start[i + 1])
        position = np.arange(r.num_computed, r.num_computed + end - at, dtype=np.int32)
        h["positions"][at:end], h["tok_seq"][at:end], h["ctx_lens"][i] = position, i, r.num_computed + end - at
        h["state"][i] = SCRATCH if r.state_slot is None else r.state_slot
        for g, group in enumerate(cache.groups):
            table = np.asarray(r.tables[g], dtype=np.int32)
            held = min(len(table), graph.max_blocks)
            h[f"tables{g}"][i] = NO_PAGE
            h[f"tables{g}"][i, :held] = table[:held]
            h[f"slots{g}"][at:end] = table[position // group.every // PAGE] * PAGE + position // group.every % PAGE
    graph._write_padding(cache, int(q_start[-1]), len(entries), len(rows))


@pytest.mark.parametrize("want", ["none", "last", "all", "some"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_description(layout, want):
    mine, theirs = make(layout, want), make(layout, want)
    assert describe(*mine) == [b + n for n, b in zip(*LAYOUTS[layout])]
    plain(*theirs)
    for name, right in theirs[0].h.items():
        assert np.array_equal(mine[0].h[name], right), name


def test_numbers_that_are_no_python_integers():
    graph, cache, entries, reqs = make("ragged prompts", "last")
    right = np.concatenate([e.tokens for e in entries])
    entries[0].tokens, entries[1].tokens, entries[2].tokens = ([np.int64(t) for t in entries[0].tokens], [float(t) for t in entries[1].tokens],
                                                              tuple(entries[2].tokens))
    describe(graph, cache, entries, reqs)
    assert np.array_equal(graph.h["tokens"][: len(right)], right)


def test_refused():
    for places, shown in (([-1], [-1]), ([32], [32]), (list(range(34)), [32, 33])):
        graph, cache, entries, reqs = make("one prompt", "last")
        entries[0].want = places
        with pytest.raises(ValueError, match=f"wanted places \\{shown}"[:-1]):
            describe(graph, cache, entries, reqs)
    for layout in ("mixed", "one prompt"):
        graph, cache, entries, reqs = make(layout, "last")
        reqs[-1].tables[0][reqs[-1].num_computed // PAGE] = NO_PAGE
        with pytest.raises(RuntimeError, match="given back"):
            describe(graph, cache, entries, reqs)


@pytest.mark.parametrize("layout, want", [("one prompt", "last"), ("one long prompt", "last"), ("one long prompt", "all"), ("behind a context", "none"),
                                          ("many single tokens", "last")])
def test_takes_no_longer_than_the_plain_lines(layout, want):
    args, best = make(layout, want), {}
    for _ in range(40):
        for f in (describe, plain):
            t0 = time.perf_counter()
            for _ in range(5):
                f(*args)
            best[f] = min(best.get(f, 1.0), time.perf_counter() - t0)
    # (32 and 33 us for the shortest prompt, 0.3 to 0.6 of the plain lines for the others; a third above them is more than the clock's noise)
    assert best[describe] <= 1.33 * best[plain], {f.__name__: f"{1e6 * t / 5:.0f} us" for f, t in best.items()}
