"""Order of the accesses to the message buffers of the chase pipeline
(evd4sc2025_b200/csrc/chase_pipe.cu), checked on the host (no GPU).

Every warp of a launch (the head, an N and an S warp per slot, the relays at the
CTA boundaries of a cooperative launch) is a sequence of tasks that wait for
messages, then write messages.  Buffers are two sweeps deep and carry no
acknowledgement, so a write is safe only if everything that reads the message
it replaces happens before it, whatever the speeds of the warps.  The test
builds that relation with vector clocks from the kernel's own conditions
(evd_test_chase_flow) and also sees that every wait ends.
"""
import ctypes as C
import pathlib
import random
import re

import pytest


def library_flow(lib):
    buf = (C.c_int * 5)()

    def flow(n, s0, s1, k, s):
        lib.evd_test_chase_flow(n, s0, s1, k, s, buf)
        return tuple(buf)
    return flow


def former_flow(n, s0, s1, k, s):
    """The rules that let a slot run its last task without waiting."""
    r = s + 1 + 32 * k
    return (min(s1 - 1, n - 2 - 32 * k), int(r <= n - 2), int(s > s0 and r + 31 <= n - 1),
            int(r + 32 <= n - 2), int(s < s1 - 1))


def programs(flow, n, s0, s1, slots_per_cta, relays):
    """{warp: [(waits, writes)]}, one entry per task in order.  A message is
    (buffer, sweep); a buffer is (kind, slot, parity)."""
    nslots = (n - 2 - s0) // 32 + 1

    def msg(kind, k, s):
        return ((kind, k, s & 1), s)

    def crosses_up(k):  # u to slot k comes from another CTA
        return relays and k > 0 and k % slots_per_cta == 0

    progs = {"head": [([msg("c", 0, s - 1), msg("cN", 0, s - 1)] if s > s0 else [],
                       [msg("u", 0, s)]) for s in range(s0, s1)]}
    for k in range(nslots):
        last = flow(n, s0, s1, k, s0)[0]
        N, S, RU, RC = [], [], [], []
        for s in range(s0, last + 1):
            _, waits_u, waits_c, sends_u, hands_row = flow(n, s0, s1, k, s)
            # a column that slot k - 1 reads across a CTA boundary goes through
            # the relay of that CTA
            cdst = "b" if crosses_up(k) else ""
            wn = [msg("u", k, s)] if waits_u else []
            ws = list(wn) + ([msg("row", k, s - 1)] if s > s0 else [])
            if waits_c:
                wn += [msg("c", k + 1, s - 1), msg("cN", k + 1, s - 1)]
                ws += [msg("c", k + 1, s - 1)]
            out_n = [msg("bu" if crosses_up(k + 1) else "u", k + 1, s)] if sends_u else []
            if s < s1 - 1:
                out_n.append(msg(cdst + "cN", k, s))
                if hands_row:
                    out_n.append(msg("row", k, s))
            N.append((wn, out_n))
            S.append((ws, [msg(cdst + "c", k, s)] if s < s1 - 1 else []))
            if waits_u and crosses_up(k):
                RU.append(([msg("bu", k, s)], [msg("u", k, s)]))
            if waits_c and crosses_up(k + 1):
                RC.append(([msg("bc", k + 1, s - 1), msg("bcN", k + 1, s - 1)],
                           [msg("c", k + 1, s - 1), msg("cN", k + 1, s - 1)]))
        progs["N", k], progs["S", k], progs["RU", k], progs["RC", k] = N, S, RU, RC
    return progs


def check(progs):
    """Runs the tasks in an order that the waits allow; returns the unordered
    overwrites and the tasks whose waits never end."""
    warps = list(progs)
    index = {w: i for i, w in enumerate(warps)}
    readers = {}
    for w in warps:
        for t, (waits, _) in enumerate(progs[w]):
            for m in waits:
                readers.setdefault(m, []).append((w, t))
    clock = {w: [0] * len(warps) for w in warps}  # tasks of each warp known to be done
    sent = {}    # message -> clock of its writer at the write
    held = {}    # buffer -> sweep of the message in it
    pos = {w: 0 for w in warps}
    bad = []
    moved = True
    while moved:
        moved = False
        for w in warps:
            while pos[w] < len(progs[w]):
                waits, writes = progs[w][pos[w]]
                if any(m not in sent for m in waits):
                    break
                clk = clock[w]
                for m in waits:
                    clk[:] = map(max, clk, sent[m])
                clk[index[w]] = pos[w] + 0.5  # this task's waits are over
                for buf, s in writes:
                    for rw, rt in readers.get((buf, held.get(buf)), ()):
                        if clk[index[rw]] < rt + 0.5:
                            bad.append((w, pos[w], buf, s, rw, rt))
                    held[buf] = s
                    sent[buf, s] = list(clk)
                pos[w] += 1
                clk[index[w]] = pos[w]
                moved = True
    stuck = [(w, pos[w]) for w in warps if pos[w] < len(progs[w])]
    return bad, stuck


CASES = [(n, 0, n - 2, 4, relays) for n in (3, 34, 35, 66, 67, 130, 131, 200, 259)
         for relays in (False, True)] + [(200, 0, 90, 4, True), (200, 90, 198, 4, True)]


@pytest.mark.parametrize("n,s0,s1,per,relays", CASES)
def test_no_message_is_overwritten_before_it_is_read(evdlib, n, s0, s1, per, relays):
    bad, stuck = check(programs(library_flow(evdlib.lib()), n, s0, s1, per, relays))
    assert not stuck and not bad, (stuck[:3], bad[:3])


def test_the_check_sees_an_unordered_last_task():
    bad, stuck = check(programs(former_flow, 131, 0, 129, 4, False))
    assert not stuck
    assert {b[2][0] for b in bad} == {"row", "c"}  # both places: the row and S's column


def test_every_bounded_wait_leaves_its_loop_as_a_whole_warp():
    """Patience::over shuffles with the full mask, so its loop may only be left
    by a vote of the warp: one loop, and every wait goes through it."""
    src = (pathlib.Path(__file__).resolve().parents[1] / "evd4sc2025_b200" / "csrc"
           / "chase_pipe.cu").read_text()
    calls = [m.start() for m in re.finditer(r"\.over\(", src)]
    assert len(calls) == 1
    loop = src[src.rindex("for (", 0, calls[0]):calls[0]]
    assert "!__all_sync(0xffffffffu, ready())" in loop


def test_the_gate_gives_every_cta_the_same_answer():
    """pass_gate: count in, then poll; out of patience, try to shut the gate on
    the number just read.  CTAs come, poll and lose patience in any order, and
    every interleaving ends with one answer, which is yes only if all came."""
    shut, ctas = 1 << 30, 5
    rng = random.Random(1)
    answers = set()
    for _ in range(4000):
        gate, read, got = 0, {}, {}
        late = rng.random() < 0.5  # some run lets patience end early
        while len(got) < ctas:
            c = rng.randrange(ctas)
            if c in got:
                continue
            if c not in read:
                gate, read[c] = gate + 1, None  # atomicAdd
            elif read[c] is None:
                v = gate  # the poll
                if v & shut:
                    got[c] = False
                elif v == ctas:
                    got[c] = True
                elif late and rng.random() < 0.3:
                    read[c] = v
            else:  # atomicCAS with the number read
                if gate == read[c]:
                    gate |= shut
                read[c] = None
        assert len(set(got.values())) == 1
        answers.add(got[0])
        assert not got[0] or gate == ctas
    assert answers == {True, False}
