"""Waits on the tensor-core correlator's operand regions (csrc/tc_steps.h),
checked over every order of events.

A warp sees the parity of a barrier's phase only: once the phase after the
awaited one has completed as well, its test answers "not yet".  The model has
the protocol's events (M1 of a step, the operand arrivals of its chain's
warps, M2, the releases of D) with two warps per chain and no timing at all,
and looks for a reachable state in which the barrier and phase that
csrc/tc_steps.h names can pass a waiting warp by.
"""
import os
import subprocess
from collections import deque

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 12  # steps
WARPS = 2  # per chain
SRC = r"""
#include <cstdio>
#include "tc_steps.h"
template <int NCH, int A2S> void print() {
  using T = tga::A2Turn<NCH, A2S>;
  for (int s = 0; s < %d; ++s)
    std::printf("%%d %%d %%d %%d %%d %%d %%u\n", NCH, A2S, (int)T::WAITS, T::REGION_BARS, T::region(s), T::bar(s), T::parity(s));
}
int main() { print<3, 2>(); print<2, 1>(); print<2, 2>(); print<3, 1>(); }
""" % N


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("steps")
    (d / "t.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.join(ROOT, "tart-gnss_b200", "csrc"), "-o", str(d / "t"),
                           str(d / "t.cpp")])
    out = {}
    for line in subprocess.check_output([str(d / "t")], text=True).splitlines():
        nch, a2s, waits, per_region, region, bar, parity = map(int, line.split())
        out.setdefault((nch, a2s), []).append((waits, per_region, region, bar, parity))
    return out


def passed_by(nch, a2s, rule):
    """The first (step, phases of the awaited barrier) found in which a wait's
    parity lies, or in which operands are stored over an M2 to come; None when
    no order of events has one."""
    wait = [r for r in rule]

    def phases(barrier, m2):  # completed phases of a region's or chain's barrier
        per_region, k = barrier
        return sum(1 for t in range(N) if m2 >> t & 1 and (wait[t][2] == k if per_region else t % nch == k))

    def awaited(s):  # barrier and number of phases that step s needs
        w, per_region, region, bar, parity = wait[s]
        if not w:
            return None
        b = (bool(per_region), bar)
        need = sum(1 for t in range(s - a2s + 1) if (wait[t][2] == bar if per_region else t % nch == bar))
        # completed phases c answer yes when their parity differs from the awaited phase's
        assert (need + 1) % 2 == parity, "parity of the phase"
        return b, need

    # state: M1s issued (in order), per (chain, warp) its progress: 2 u + (0:
    # before storing operands of its use u, 1: stored, before its M2); M2s done
    start = (0, (0,) * (nch * WARPS), 0)
    seen, todo = {start}, deque([start])
    while todo:
        m1, prog, m2 = todo.popleft()
        nxt = []
        stored = [0] * N
        freed = [0] * N
        for i, p in enumerate(prog):
            x = i // WARPS
            for u in range(p // 2 + 1):
                s = u * nch + x
                if s < N:
                    stored[s] += p >= 2 * u + 1
                    freed[s] += p >= 2 * u + 2
        # M1 of step s: D free of step s - nch
        if m1 < N and (m1 < nch or freed[m1 - nch] == WARPS):
            nxt.append((m1 + 1, prog, m2))
        for s in range(N):
            if stored[s] == WARPS and not m2 >> s & 1:
                nxt.append((m1, prog, m2 | 1 << s))
        for i, p in enumerate(prog):
            s = p // 2 * nch + i // WARPS
            if s >= N:
                continue
            go = prog[:i] + (p + 1,) + prog[i + 1:]
            if p % 2 == 0:
                a = awaited(s)
                if a is not None:
                    c = phases(a[0], m2)
                    if c > a[1]:
                        return s, c
                    free = c == a[1]
                else:
                    free = True
                if m1 > s and free:
                    if s >= a2s and not m2 >> (s - a2s) & 1:
                        return s, "stored over operands in use"
                    nxt.append((m1, go, m2))
            elif m2 >> s & 1:
                nxt.append((m1, go, m2))
        for t in nxt:
            if t not in seen:
                seen.add(t)
                todo.append(t)
    return None


@pytest.mark.parametrize("nch,a2s", [(3, 2), (2, 1), (2, 2), (3, 1)])
def test_no_phase_passes_a_waiting_warp(rules, nch, a2s):
    assert passed_by(nch, a2s, rules[(nch, a2s)]) is None


def test_the_model_sees_a_phase_passed_by():
    """Three chains on two regions with the M2 barrier of step s - 2's chain:
    the phase that step s + 1 completes does not wait for step s's warps."""
    nch, a2s = 3, 2
    rule = [(1, 0, s % a2s, (s - a2s) % nch, (s + nch - a2s) // nch + 1 & 1) for s in range(N)]
    assert passed_by(nch, a2s, rule) is not None
