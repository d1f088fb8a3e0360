"""The exchange of the one-launch coarsest solve (k_coarse_solve), as a model
whose schedules are all visited: two CTAs, each with a thread that owns the
cells on the cut (and arms the mbarriers) and one that owns none.

A pass is: update and send, block barrier, wait for the other CTA's values of
the colour by the parity of that colour's mbarrier.  The cluster barrier is
arrived at after a black pass and waited for after the next red one.  The
mbarrier of a colour carries one phase per sweep; a phase completes once it is
armed (its bytes expected) and its bytes are in, and a wait by parity sees the
phase it waits for only until the next one completes.

Armed right behind the arming thread's own wait, a phase can complete while
the other thread has yet to look at the one before: that thread, and with it
the cluster, stops.  Armed behind the next block barrier, where the kernel
does it, every schedule ends.
"""
import pytest

SWEEPS = 3


def _steps(arm):
    """Statements of a thread's passes: (kind, colour, sweep)."""
    out = []
    for sw in range(SWEEPS):
        for col in (0, 1):
            out.append(("send", col, sw))
            out.append(("block", col, sw))
            if arm == "behind the block barrier" and (col == 1 or sw > 0):
                out.append(("arm", 1 - col, sw))
            if col == 1:
                out.append(("arrive", col, sw))
            out.append(("wait", col, sw))
            if arm == "behind the wait":
                out.append(("arm", col, sw))
            if col == 0 and sw > 0:
                out.append(("cluster", col, sw))
    return out


def _settle(bar):
    """(phase, armed, bytes in) with the phase completed where it can be."""
    phase, armed, got = bar
    return (phase + 1, 0, got - 1) if armed and got >= 1 else bar


def _moves(state, prog):
    """Successors of a state: program counters of the four threads (two per
    CTA, the first owns the cut), mbarriers per CTA and colour, values in
    flight per CTA and colour, cluster arrivals per thread."""
    pcs, bars, fly, arrived = state
    for t in range(4):
        if pcs[t] == len(prog):
            continue
        cta, owner = divmod(t, 2)
        kind, col, sw = prog[pcs[t]]
        npc = list(pcs)
        nbars, nfly, narr = list(bars), list(fly), list(arrived)
        at = 2 * cta + col
        npc[t] += 1
        if kind == "send":
            if owner == 0:
                nfly[2 * (1 - cta) + col] += 1
        elif kind == "block":
            # passes once the other thread of the CTA is at this barrier too
            # (or beyond it)
            if pcs[t ^ 1] < pcs[t]:
                continue
        elif kind == "arm":
            if owner == 0:
                phase, armed, got = bars[at]
                assert not armed, "armed twice"
                nbars[at] = _settle((phase, 1, got))
        elif kind == "arrive":
            narr[t] += 1
        elif kind == "wait":
            if (bars[at][0] & 1) == (sw & 1):
                continue  # by parity: not complete, as far as the thread can tell
        elif kind == "cluster":
            if min(arrived) < sw:
                continue
        yield tuple(npc), tuple(nbars), tuple(nfly), tuple(narr)
    for at in range(4):
        if fly[at]:
            nfly, nbars = list(fly), list(bars)
            nfly[at] -= 1
            phase, armed, got = bars[at]
            # no value lands while the owner's update of the other colour has
            # yet to read the one before
            cta, col = divmod(at, 2)
            landed = phase + got  # sweep of this value
            if landed > 0:
                reader = prog.index(("send", 1 - col, landed - 1 + col))
                assert pcs[2 * cta] > reader, "a copy is overwritten before it is read"
            nbars[at] = _settle((phase, armed, got + 1))
            yield pcs, tuple(nbars), tuple(nfly), arrived


def _stuck(arm):
    """States from which nothing moves and not every thread is done."""
    prog = _steps(arm)
    first = ((0,) * 4, ((0, 1, 0),) * 4, (0,) * 4, (0,) * 4)
    seen, todo, stuck = {first}, [first], []
    while todo:
        s = todo.pop()
        nxt = list(_moves(s, prog))
        if not nxt and any(pc != len(prog) for pc in s[0]):
            stuck.append(s)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return stuck, prog


def test_every_schedule_ends():
    stuck, _ = _stuck("behind the block barrier")
    assert not stuck


def test_arming_behind_the_wait_strands_a_late_thread():
    stuck, prog = _stuck("behind the wait")
    assert stuck
    # a thread without cells on the cut, at its wait for a phase that completed
    assert any(prog[pc][0] == "wait" and bars[2 * (t // 2) + prog[pc][1]][0] > prog[pc][2]
               for pcs, bars, *_ in stuck for t, pc in enumerate(pcs)
               if t % 2 and pc < len(prog))
