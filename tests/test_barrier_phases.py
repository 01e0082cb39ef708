"""Barrier phases of the dQ kernels, on the CPU.

A wait on an mbarrier names a phase by its parity, so a waiter must never be two phases behind: the phase it waits for would look
as if it had not come yet, and never come again. The roles of a kernel are written down here as the waits and arrivals they
make; for every wait of every role, that role is held there while all others run as far as they can.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dark-forest_b200", "csrc")


class Role(list):
    """The waits and arrivals of one role in order; copies, loads and products count as done at once, the worst case here."""

    def wait(self, bar, phase):
        self.append(("wait", bar, phase))

    def arrive(self, bar):
        self.append(("arrive", bar, 0))


def dq_tf32(items, ds_bars):
    """k_attn_bwd_dq_tf32_d64 for a CTA with items of that many key tiles; two threads stand for the compute warps."""
    load_k, load_m, mma, compute = Role(), Role(), Role(), Role()
    steps = [(n, j) for n, n_kv in enumerate(items) for j in range(n_kv)]
    last = [j + 1 == items[n] for n, j in steps]
    for g, (n, j) in enumerate(steps):
        if j == 0:
            if n > 0:
                load_k.wait("Q_EMPTY", n - 1)
            load_k.arrive("Q_FULL")
        if g > 0:
            load_k.wait("S_FULL", g - 1)
            load_m.wait("KM_EMPTY", g - 1)
        load_k.arrive("KK_FULL")
        if j == 0:
            if n > 0:
                load_k.wait("G_EMPTY", n - 1)
                load_k.wait("O_FREE", n - 1)
            load_k.arrive("GO_FULL")
        if g > 0:
            load_k.wait("DP_FULL%d" % ((g - 1) % 2), (g - 1) // 2)
        load_k.arrive("VK_FULL")
        load_m.arrive("KM_FULL")
        if last[g]:
            load_m.wait("EPI_FULL", n)

    def scores(g):
        mma.wait("KK_FULL", g)
        mma.arrive("S_FULL")
        if last[g]:
            mma.arrive("Q_EMPTY")

    def dp(g):
        mma.wait("VK_FULL", g)
        mma.arrive("DP_FULL%d" % (g % 2))
        if last[g]:
            mma.arrive("G_EMPTY")

    mma.wait("Q_FULL", 0)
    scores(0)
    mma.wait("GO_FULL", 0)
    dp(0)
    for g, (n, j) in enumerate(steps):
        more = g + 1 < len(steps)
        if more:
            mma.wait("S_FREE", g)
            if last[g]:
                mma.wait("Q_FULL", n + 1)
            scores(g + 1)
            if not last[g]:
                dp(g + 1)
        mma.wait("DS_FULL%d" % (g % ds_bars), g // ds_bars)
        mma.wait("KM_FULL", g)
        mma.arrive("KM_EMPTY")
        if last[g]:
            mma.arrive("ACC_FULL")
        if more and last[g]:
            mma.wait("GO_FULL", n + 1)
            dp(g + 1)

    def row_sums(n):
        compute.wait("GO_FULL", n)
        compute.arrive("O_FREE")
        compute.arrive("DX_FULL")
        compute.wait("DX_FULL", n)

    row_sums(0)
    for g, (n, j) in enumerate(steps):
        compute.wait("S_FULL", g)
        compute.arrive("S_FREE")
        compute.wait("DP_FULL%d" % (g % 2), g // 2)
        compute.arrive("DS_FULL%d" % (g % ds_bars))
        if last[g]:
            if n + 1 < len(items):
                row_sums(n + 1)
            compute.wait("ACC_FULL", n)
            compute.arrive("EPI_FULL")
    return {"load_k": load_k, "load_m": load_m, "mma": mma, "compute 0": compute, "compute 1": compute}


def phases_missed(roles):
    """(role, barrier, phase) of every wait that can find its barrier two phases on; fails when a role does not reach its end."""
    counts = {}
    for name, role in roles.items():
        for op, bar, _ in role:
            if op == "arrive":
                counts.setdefault(bar, set()).add(name)

    def run(held=None, at=None):
        pos, arrived = dict.fromkeys(roles, 0), dict.fromkeys(counts, 0)
        moved = True
        while moved:
            moved = False
            for name, role in roles.items():
                while pos[name] < len(role) and not (name == held and pos[name] == at):
                    op, bar, phase = role[pos[name]]
                    if op == "wait" and arrived[bar] // len(counts[bar]) <= phase:
                        break
                    if op == "arrive":
                        arrived[bar] += 1
                    pos[name] += 1
                    moved = True
        return pos, {b: arrived[b] // len(counts[b]) for b in counts}

    pos, _ = run()
    assert all(pos[name] == len(role) for name, role in roles.items()), pos
    missed = []
    for name, role in roles.items():
        for at, (op, bar, phase) in enumerate(role):
            if op == "wait" and run(name, at)[1][bar] > phase + 1:
                missed.append((name, bar, phase))
    return missed


def test_one_barrier_for_two_buffers_is_missed():
    assert {m[:2] for m in phases_missed(dq_tf32([4], 1))} == {("mma", "DS_FULL0")}


@pytest.mark.parametrize("items", [[1], [2], [1, 1, 1], [5, 2, 1, 3], [7, 6]])
def test_tf32_dq_waits_see_every_phase(items):
    with open(os.path.join(CSRC, "attn_bwd_sm100.cu")) as f:
        enum = re.search(r"namespace dq \{\s*enum Bar \{(.*?)\}", f.read(), re.S).group(1)
    ds_bars = len(re.findall(r"\bDS_FULL\d?\b", enum))
    assert phases_missed(dq_tf32(items, ds_bars)) == []
