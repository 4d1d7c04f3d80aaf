"""The order that the barriers of the tcgen05 prompt attention enforce, over all interleavings of its warps.

Softmax warps write P of a tile into one of two buffers and announce it; the MMA warp issues the next tile's scores and,
when P is announced, P V, which the tensor cores finish in order.  A warp whose maxima stay waits for P V of two tiles
before, one whose maxima move for P V of the tile before, so warps may be a tile apart.  Waits go by parity, as the
hardware's do."""
import re
from pathlib import Path

import pytest

import zinfer_b200.csrc

SOURCE = Path(zinfer_b200.csrc.__file__).parent / "attention_prefill_tc5.cu"


def announce_barriers():
    """Barriers that "P is written" goes over in the kernel: tile t's is number t mod that."""
    text = SOURCE.read_text()
    n = re.search(r"constexpr int NP = (\d+);", text)
    per_buffer = "mbar_arrive(&p_ready[t % NP])" in text and "mbar_wait(&p_ready[t % NP], (t / NP) & 1)" in text
    return int(n.group(1)) if n and per_buffer else 1


def faults(warps, tiles, barriers):
    """What some interleaving does wrong.  A state: (next tile and stage of the MMA warp, operations the tensor cores have not
    finished, per softmax warp its tile, stage and whether its maximum moved, completed phases of the score barriers,
    (phases, arrivals) per announcing barrier, completed phases of the P V barriers, P V issued, P V finished)."""
    passed = lambda phases, phase: (phases & 1) != (phase & 1)
    at = lambda seq, i, v: seq[:i] + (v,) + seq[i + 1:]
    first = (-1, 0), (), ((0, 0, 0),) * warps, (0, 0), ((0, 0),) * barriers, (0, 0), 0, 0
    seen, todo, wrong = {first}, [first], set()
    while todo:
        mma, queue, ws, s_full, ready, pv, issued, finished = state = todo.pop()
        after = []

        def go(mma=mma, queue=queue, ws=ws, s_full=s_full, ready=ready, pv=pv, issued=issued, finished=finished):
            after.append((mma, queue, ws, s_full, ready, pv, issued, finished))

        def scores(t):
            if any(w[0] < t - 2 or (w[0] == t - 2 and w[1] < 2) for w in ws):
                wrong.add("scores overwritten before they are read")
            return queue + (("S", t),)

        if queue:
            op, t = queue[0]
            if op == "S":
                go(queue=queue[1:], s_full=at(s_full, t & 1, s_full[t & 1] + 1))
            else:
                go(queue=queue[1:], pv=at(pv, t & 1, pv[t & 1] + 1), finished=finished + 1)
        t, stage = mma
        if t == -1:
            go(mma=(0, 0), queue=scores(0))
        elif t < tiles and stage == 0:
            go(mma=(t, 1), queue=scores(t + 1) if t + 1 < tiles else queue)
        elif t < tiles and passed(ready[t % barriers][0], t // barriers):
            if any(w[0] <= t for w in ws):
                wrong.add("P V begins before a warp has announced its rows of P")
            go(mma=(t + 1, 0), queue=queue + (("P", t),), issued=issued + 1)
        for i, (t, stage, moved) in enumerate(ws):
            if t == tiles:
                continue
            if stage == 0 and passed(s_full[t & 1], t >> 1):
                go(ws=at(ws, i, (t, 1, 0)))
            elif stage == 1:
                if s_full[t & 1] != (t >> 1) + 1:
                    wrong.add("another tile's scores are read")
                go(ws=at(ws, i, (t, 2, 0)))
                go(ws=at(ws, i, (t, 2, 1)))
            elif stage == 2:
                need = t - 1 if moved else t - 2
                if need < 0 or passed(pv[need & 1], need >> 1):
                    if need >= finished:
                        wrong.add("a wait for P V passes too early")
                    go(ws=at(ws, i, (t, 3, moved)))
            elif stage == 3:
                if t > 0 and moved and issued != finished:
                    wrong.add("O is rescaled while P V adds to it")
                if ("P", t - 2) in queue:
                    wrong.add("P is overwritten while P V reads it")
                phases, arrived = ready[t % barriers]
                now = (phases + 1, 0) if arrived + 1 == warps else (phases, arrived + 1)
                go(ws=at(ws, i, (t + 1, 0, 0)), ready=at(ready, t % barriers, now))
        if not after and not (mma[0] == tiles and not queue and all(w[0] == tiles for w in ws)):
            wrong.add("all wait")
        for nxt in after:
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
    return wrong


@pytest.mark.parametrize("warps,tiles", [(1, 7), (2, 7), (3, 6), (4, 4)])
def test_no_interleaving_of_the_warps_breaks_the_order(warps, tiles):
    assert faults(warps, tiles, announce_barriers()) == set()


def test_one_barrier_for_both_buffers_would_break_it():
    assert "P V begins before a warp has announced its rows of P" in faults(2, 4, 1)
