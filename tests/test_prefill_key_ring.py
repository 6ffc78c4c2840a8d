"""The key ring of the prefill attention kernel, as a model on the CPU: one producer, two score issuers that take alternate
tiles, copies that land in any order. Every interleaving of the first tiles is walked. An issuer must only ever pass its wait
for a tile that has landed, and a barrier must never be armed twice in one phase (on the device: an arrival that no phase
expects, which ends the kernel). Ring and barrier counts are the kernel's, read from its source."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cwick_b200", "csrc", "mla_prefill_attn.cu")


def passes(done, parity):
    """mbarrier.try_wait.parity on a barrier with `done` completed phases: only the parity of the pending one is known."""
    return done & 1 != parity


def walk(slots, bars, tiles):
    """A fault as text, or None. State: tiles armed by the producer; per barrier (completed phases, tile on its way or -1); per
    slot completed "empty" phases; each issuer's next tile; per score buffer the tile in it or -1; each softmax pair's next tile to load
    and the tile it holds (-1: none) until its P may be written; value products done; P tiles written."""
    start = (0, ((0, -1),) * bars, (0,) * slots, (0, 1), (-1, -1), (0, 1), (-1, -1), 0, frozenset())
    seen, todo = {start}, [start]
    while todo:
        armed, full, empty, nxt, score, load, held, value, written = todo.pop()
        out = []

        def put(t, i, v):
            return t[:i] + (v,) + t[i + 1:]
        if armed < tiles and passes(empty[armed % slots], (armed // slots & 1) ^ 1):
            b = armed % bars
            if full[b][1] >= 0:
                return "tile %d: barrier %d armed while tile %d is on its way" % (armed, b, full[b][1])
            out.append((armed + 1, put(full, b, (full[b][0], armed)), empty, nxt, score, load, held, value, written))
        for b, (done, tile) in enumerate(full):
            if tile >= 0:                                               # a copy lands
                out.append((armed, put(full, b, (done + 1, -1)), empty, nxt, score, load, held, value, written))
        for q in (0, 1):
            kc = nxt[q]
            if kc < tiles and score[q] < 0 and passes(full[kc % bars][0], kc // bars & 1):
                if kc >= armed or full[kc % bars][1] == kc:
                    return "tile %d: scores before its keys are here" % kc
                out.append((armed, full, put(empty, kc % slots, empty[kc % slots] + 1), put(nxt, q, kc + 2), put(score, q, kc), load, held, value, written))
            if score[q] == load[q] and held[q] < 0:                     # the pair takes the scores and frees the buffer
                out.append((armed, full, empty, nxt, put(score, q, -1), put(load, q, load[q] + 2), put(held, q, load[q]), value, written))
            if held[q] >= 0 and value > held[q] - 2:                    # P goes where the value product of two tiles ago has read
                out.append((armed, full, empty, nxt, score, load, put(held, q, -1), value, written | {held[q]}))
        if value in written:
            out.append((armed, full, empty, nxt, score, load, held, value + 1, written - {value}))
        if not out and value < tiles:
            return "stuck at value product %d" % value
        for s in out:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_the_kernels_ring():
    text = open(SRC).read()
    slots = int(re.search(r"PA_KST = (\d+);", text)[1])
    m = re.search(r"PA_KBAR = (?:(\d+) \* PA_KST|PA_KST|(\d+));", text)
    bars = slots if m is None else slots * int(m[1]) if m[1] else int(m[2] or slots)
    assert walk(slots, bars, 3 * bars + 1) is None


@pytest.mark.parametrize("slots,bars,fine", [(3, 3, False), (3, 6, True), (2, 2, True), (4, 4, True), (5, 5, False)])
def test_the_model_tells_rings_apart(slots, bars, fine):
    assert (walk(slots, bars, 9) is None) == fine
