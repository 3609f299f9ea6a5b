"""The barriers of the tcgen05 skinny GEMM (k_gemm3), without a GPU: the operations of all agents of a CTA (the kernel's own walk and
numbering), run together with vector clocks.

A wait names a phase by its parity only, so it is right only if the waiter KNOWS that the phase before has completed (else that one's
pending parity reads as the wanted phase complete) and if the phase behind cannot complete before the waiter has looked.  Copies and MMAs
complete in any order: an arrival by one of them knows what its issuer knew, nothing else."""
import ctypes as C

import pytest

WAIT, ARRIVE, LATER = 0, 1, 2


def _traces(L, nc, nsl, tiles):
    groups = 2 if nc == 32 else 3
    out = []
    for agent in range(2 * groups + 1):
        n = L.llb_b200_gemm3_trace(nc, nsl, tiles, agent, (C.c_int * 3)(), 0)
        if n < 0:
            return None
        buf = (C.c_int * (3 * n))()
        assert L.llb_b200_gemm3_trace(nc, nsl, tiles, agent, buf, 3 * n) == n
        ops = [tuple(buf[3 * i:3 * i + 3]) for i in range(n)]
        out += [ops] * (4 if agent < groups else 1)       # a group is four warps, each an agent
    return out


def _join(a, b):
    for i, v in enumerate(b):
        if v > a[i]:
            a[i] = v


def check(traces, count):
    """None, or what is wrong with these agents' operations on barriers whose phases take count[b] arrivals."""
    na, nb = len(traces), len(count)
    clock = [[0] * na for _ in range(na)]                 # clock[a]: what agent a knows of every agent's time ...
    known = [[0] * nb for _ in range(na)]                 # ... and how many phases of every barrier it knows to be complete
    pend = [[0, [0] * na, [0] * nb] for _ in range(nb)]   # arrivals of the phase in progress and what they know
    done = [[] for _ in range(nb)]                        # completed phases: what a waiter learns
    seen = [[] for _ in range(nb)]                        # per completed phase: (agent, time) of those who waited for it
    at = [0] * na
    while True:
        moved = False
        for a in range(na):
            while at[a] < len(traces[a]):
                kind, b, v = traces[a][at[a]]
                if kind == WAIT:
                    if len(done[b]) <= v:
                        break
                    if known[a][b] < v:
                        return f"agent {a} waits for phase {v} of barrier {b}, knowing of {known[a][b]} complete ones"
                    if len(done[b]) > v + 1:
                        return f"phase {v + 1} of barrier {b} completed before agent {a} had looked for phase {v}"
                    _join(clock[a], done[b][v][0])
                    _join(known[a], done[b][v][1])
                    clock[a][a] += 1
                    seen[b][v].append((a, clock[a][a]))
                else:
                    clock[a][a] += 1
                    pend[b][0] += v
                    _join(pend[b][1], clock[a])
                    _join(pend[b][2], known[a])
                    if pend[b][0] > count[b]:
                        return f"barrier {b} got {pend[b][0]} of {count[b]} arrivals"
                    if pend[b][0] == count[b]:
                        p = len(done[b])
                        if p and any(pend[b][1][w] < t for w, t in seen[b][p - 1]):
                            return f"phase {p} of barrier {b} may complete before all have looked for phase {p - 1}"
                        pend[b][2][b] = p + 1
                        done[b].append((pend[b][1], pend[b][2]))
                        seen[b].append([])
                        pend[b] = [0, [0] * na, [0] * nb]
                at[a] += 1
                moved = True
        if all(i == len(t) for i, t in zip(at, traces)):
            return None
        if not moved:
            return "nobody can go on: " + str([t[i] for i, t in zip(at, traces) if i < len(t)])


@pytest.mark.parametrize("nc", [8, 16, 32])
def test_no_wait_takes_one_phase_for_another(pkg, nc):
    L = pkg.llb.lib()
    count = []
    while L.llb_b200_gemm3_bar_count(nc, len(count)) > 0:
        count.append(L.llb_b200_gemm3_bar_count(nc, len(count)))
    ran = 0
    for nsl in range(1, 80):
        traces = _traces(L, nc, nsl, 9)
        if traces is not None:
            assert check(traces, count) is None, nsl
            ran += 1
    assert ran >= (22, 11, 6)[(8, 16, 32).index(nc)]


def test_the_check_finds_a_phase_taken_for_another():
    """Two copies into one stage, a reader that passes over the first: with one barrier it may take the first one's parity."""
    producer = [(LATER, 0, 1), (LATER, 1, 1), (WAIT, 2, 0), (LATER, 0, 1)]
    other = [(WAIT, 0, 0), (ARRIVE, 2, 1), (WAIT, 0, 1)]
    passes_over = [(WAIT, 1, 0), (WAIT, 0, 1)]
    assert "knowing of 0 complete" in check([producer, other, passes_over], [1, 1, 1])
    assert check([producer, other, [(WAIT, 1, 0), (WAIT, 0, 0)]], [1, 1, 1]) is not None     # it may come too late for the first
    assert check([producer, other], [1, 1, 1]) is None
