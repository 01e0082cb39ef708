"""Barrier phases of the backward kernels and of the split fp32 kernels, on the CPU.

A wait on an mbarrier names a phase by its parity, so a waiter must never be two phases behind: the phase it waits for would look
as if it had not come yet, and never come again. Nor may it come two phases early: the phase before the last would pass for the one it
waits for. The roles of a kernel are written down here as the waits and arrivals they make; for every wait of every role, that role is held
there while all others run as far as they can, and for every arrival the arriving role is held ahead of it. Places that no barrier of their own
guards (row statistics) are marked where they are written and read, and roles are held at the marks.
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

    def mark(self, what, k):
        self.append(("mark", what, k))


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


def dq_bf16(n_kv, ds_bars, ring=4):
    """k_attn_bwd_dq_bf16 with two issuing warps (head dimension 64)."""
    load_k, load_v, scores, dp_dq, compute = Role(), Role(), Role(), Role(), Role()
    for j in range(n_kv):
        for role, tile in ((load_k, "K"), (load_v, "V")):
            if j >= ring:
                role.wait("%s_EMPTY%d" % (tile, j % ring), j // ring - 1)
            role.arrive("%s_FULL%d" % (tile, j % ring))
        scores.wait("K_FULL%d" % (j % ring), j // ring)
        if j > 0:
            scores.wait("S_FREE", j - 1)
        scores.arrive("S_FULL")

    def dp(j):
        dp_dq.wait("V_FULL%d" % (j % ring), j // ring)
        dp_dq.arrive("DP_FULL%d" % (j % 2))
        dp_dq.arrive("V_EMPTY%d" % (j % ring))

    dp(0)
    for j in range(n_kv):
        if j + 1 < n_kv:
            dp(j + 1)
        dp_dq.wait("K_FULL%d" % (j % ring), j // ring)
        dp_dq.wait("DS_FULL%d" % (j % ds_bars), j // ds_bars)
        dp_dq.arrive("K_EMPTY%d" % (j % ring))
        compute.wait("S_FULL", j)
        compute.arrive("S_FREE")
        compute.wait("DP_FULL%d" % (j % 2), j // 2)
        compute.arrive("DS_FULL%d" % (j % ds_bars))
    dp_dq.arrive("ACC_FULL")
    compute.wait("ACC_FULL", 0)
    return {"load_k": load_k, "load_v": load_v, "scores": scores, "dp_dq": dp_dq, "compute 0": compute, "compute 1": compute}


def dkdv_tf32(items):
    """k_attn_bwd_dkdv_tf32_d64 for a CTA with items of that many query tiles: each group of compute warps has half of a step's queries."""
    load_k, load_m = Role(), Role()
    steps = [(n, i) for n, n_it in enumerate(items) for i in range(n_it)]
    last = [i + 1 == items[n] for n, i in steps]
    first_tile = [sum(items[:n]) + n for n in range(len(items) + 1)]  # of an item in the rings: its K (V)
    for r in range(first_tile[-1]):
        for tile in ("QK", "GK"):
            if r > 1:
                load_k.wait("%s_EMPTY%d" % (tile, r % 2), r // 2 - 1)
            load_k.arrive("%s_FULL%d" % (tile, r % 2))
    for g, (n, i) in enumerate(steps):
        for tile in ("GM", "QM"):
            for h in range(2):
                if g > 0:
                    load_m.wait("%s_EMPTY%d" % (tile, h), g - 1)
                load_m.arrive("%s_FULL%d" % (tile, h))
        if last[g]:
            load_m.wait("EPI_FULL", n)

    moved = [sum(n_it > 1 for n_it in items[:n]) for n in range(len(items) + 1)]  # items before whose K and V went to tensor memory

    def chain(ring, kv, scores, ready, tile):
        role = Role()

        def first(h, r, frees):
            if h == 0:
                role.wait("%s_FULL%d" % (ring, r % 2), r // 2)
            if h == 0 and r == 1:
                role.wait("FIRST", 0)
            role.arrive("%s%d" % (scores, h))
            if h == 1:
                role.arrive("%s_EMPTY%d" % (ring, r % 2))
                if frees:
                    role.arrive(kv + "_FREE")

        g = 0
        for n, n_it in enumerate(items):
            r = first_tile[n]
            role.wait("%s_FULL%d" % (ring, r % 2), r // 2)
            first(0, r + 1, False)
            first(1, r + 1, False)
            if n_it > 1:
                role.wait(kv + "_READY", moved[n])
            role.arrive("%s_EMPTY%d" % (ring, r % 2))
            for i in range(n_it):
                for h in range(2):
                    role.wait("%s%d" % (ready, h), g)
                    role.wait("%s_FULL%d" % (tile, h), g)
                    role.arrive("%s_EMPTY%d" % (tile, h))
                    if i + 1 == n_it and h == 1:
                        role.arrive("ACC_FULL")
                    if i + 1 < n_it:
                        first(h, r + 2 + i, i + 2 == n_it)
                g += 1
        return role

    def group(h):
        role = Role()

        def resident(ring, kv, n):
            if n < len(items) and items[n] > 1:
                if moved[n] > 0:
                    role.wait(kv + "_FREE", moved[n] - 1)
                role.wait("%s_FULL%d" % (ring, first_tile[n] % 2), first_tile[n] // 2)
                role.arrive(kv + "_READY")

        role.arrive("FIRST")
        resident("QK", "K", 0)
        for g, (n, i) in enumerate(steps):
            role.wait("S_FULL%d" % h, g)
            role.arrive("P_FULL%d" % h)
            if last[g]:
                resident("QK", "K", n + 1)
            elif g == 0:
                resident("GK", "V", 0)
            role.wait("DP_FULL%d" % h, g)
            role.arrive("DS_FULL%d" % h)
            if last[g]:
                resident("GK", "V", n + 1)
                role.wait("ACC_FULL", n)
                role.arrive("EPI_FULL")
        return role

    roles = {"load_k": load_k, "load_m": load_m, "s_dv": chain("QK", "K", "S_FULL", "P_FULL", "GM"),
             "dp_dk": chain("GK", "V", "DP_FULL", "DS_FULL", "QM")}
    for h in range(2):
        for x in "ab":
            roles["group %d %s" % (h, x)] = group(h)
    return roles


def dkdv_bf16(n_it, issuers, s_bufs, ring=4):
    """k_attn_bwd_dkdv_bf16: two issuing warps and two S^T buffers (head dimension 64), or one of each (128); two threads stand for each half of the
    compute warps, the one that stages lse and the one that stages delta."""
    load_q, load_g, chains = Role(), Role(), [Role() for _ in range(issuers)]
    for it in range(n_it):
        for role, tile in ((load_q, "Q"), (load_g, "G")):
            if it >= ring:
                role.wait("%s_EMPTY%d" % (tile, it % ring), it // ring - 1)
            role.arrive("%s_FULL%d" % (tile, it % ring))

    def scores(role, chain_s, it):
        tile = "Q" if chain_s else "G"
        role.wait("%s_FULL%d" % (tile, it % ring), it // ring)
        if it < s_bufs:
            role.wait("FIRST", 0)
        role.mark("lse used" if chain_s else "delta used", it)
        role.arrive("S_FULL%d" % (it % s_bufs) if chain_s else "DP_FULL")
        if issuers == 2:
            role.arrive("%s_EMPTY%d" % (tile, it % ring))

    def gradient(role, chain_s, it):
        tile = "G" if chain_s else "Q"
        if issuers == 2:
            role.wait("%s_FULL%d" % (tile, it % ring), it // ring)
        role.wait("P_FULL%d" % (it % s_bufs), it // s_bufs) if chain_s else role.wait("DS_FULL", it)
        role.arrive("%s_EMPTY%d" % (tile, it % ring))

    if issuers == 2:
        for role, chain_s in zip(chains, (True, False)):
            ahead = s_bufs if chain_s else 1
            for it in range(min(ahead, n_it)):
                scores(role, chain_s, it)
            for it in range(n_it):
                gradient(role, chain_s, it)
                if it + ahead < n_it:
                    scores(role, chain_s, it + ahead)
    else:
        scores(chains[0], True, 0)
        scores(chains[0], False, 0)
        for it in range(n_it):
            for chain_s in (True, False):
                gradient(chains[0], chain_s, it)
                if it + 1 < n_it:
                    scores(chains[0], chain_s, it + 1)
    for role in chains:
        role.arrive("ACC_FULL")

    def half(lse):
        role, ahead, stat = Role(), s_bufs if lse else 1, "lse" if lse else "delta"
        for it in range(min(ahead, n_it)):
            role.mark(stat + " staged", it)
        role.arrive("FIRST")
        for it in range(n_it):
            more = it + ahead < n_it
            role.wait("S_FULL%d" % (it % s_bufs), it // s_bufs)
            if lse and more:
                role.mark("lse staged", it + ahead)
            role.arrive("P_FULL%d" % (it % s_bufs))
            role.wait("DP_FULL", it)
            if not lse and more:
                role.mark("delta staged", it + ahead)
            role.arrive("DS_FULL")
        role.wait("ACC_FULL", 0)
        return role

    roles = {"load_q": load_q, "load_g": load_g, **{"issuer %d" % i: role for i, role in enumerate(chains)}}
    roles.update({"%s %s" % (name, x): half(name == "lse") for name in ("lse", "delta") for x in "ab"})
    return roles


def split(n, two, keys, st2):
    """split_block of attn_split_sm100.cu with n steps. two: DQ and DK, else FORWARD and DV; keys: resident rows are keys (DK, DV), whose steps bring
    row statistics; st2: buffers of the second streamed tile. Two threads stand for the streaming warps, two for the compute warps."""
    def stage2(j):
        return j % st2, j // st2

    def stream():
        role = Role()
        for j in range(n):
            for tile, (st, use) in (("B1", (j % 2, j // 2)), ("B2", stage2(j))):
                if use > 0:
                    role.wait("%s_EMPTY%d" % (tile, st), use - 1)
                role.arrive("%s_FULL%d" % (tile, st))
        return role

    mma = Role()

    def scores(j):
        mma.wait("B1_FULL%d" % (j % 2), j // 2)
        if j > 0:
            mma.wait("R_FREE" if two else "S_FREE", j - 1)
        mma.arrive("S_FULL0" if two else "S_FULL%d" % (j % 2))
        if not two:
            mma.arrive("B1_EMPTY%d" % (j % 2))

    def dp(j):
        st, use = stage2(j)
        mma.wait("B2_FULL%d" % st, use)
        mma.arrive("DP_FULL")
        mma.arrive("B2_EMPTY%d" % st)

    def result(j):
        st, use = stage2(j)
        if two:
            mma.wait("T_FULL0", j)
            mma.wait("T_FULL1", j)
        else:
            mma.wait("T_FULL%d" % (j % 2), j // 2)
            mma.wait("B2_FULL%d" % st, use)
            if j > 0:
                mma.wait("R_FREE", j - 1)
        mma.arrive("R_FULL")
        mma.arrive("B1_EMPTY%d" % (j % 2) if two else "B2_EMPTY%d" % st)

    mma.wait("A_READY", 0)
    scores(0)
    for j in range(n):
        if two:
            dp(j)
            result(j)
        if j + 1 < n:
            scores(j + 1)
        if not two:
            result(j)

    def compute():
        role = Role()

        def add_r(j):
            role.wait("R_FULL", j)
            role.arrive("R_FREE")

        def stats(j):
            role.mark("stats written", j)
            role.arrive("STAT_FULL")

        role.arrive("A_READY")
        if keys:
            stats(0)
        for j in range(n):
            if two and j > 0:
                add_r(j - 1)
            if keys:
                role.wait("STAT_FULL", j)
            role.wait("S_FULL0" if two else "S_FULL%d" % (j % 2), j if two else j // 2)
            if not two:
                role.arrive("S_FREE")
            else:
                role.wait("DP_FULL", j)
            if keys:
                role.mark("stats read", j)
            for x in (0, 1) if two else (j % 2,):
                role.arrive("T_FULL%d" % x)
            if keys and j + 1 < n:
                stats(j + 1)
            if not two and j > 0:
                add_r(j - 1)
        add_r(n - 1)
        return role

    return {"stream 0": stream(), "stream 1": stream(), "mma": mma, "compute 0": compute(), "compute 1": compute()}


def _runner(roles):
    counts = {}
    for name, role in roles.items():
        for op, bar, _ in role:
            if op == "arrive":
                counts.setdefault(bar, set()).add(name)

    def run(held=None, at=None):
        """Everybody as far as they can, `held` not past its entry `at`: positions and completed phases."""
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

    return run


def phases_missed(roles):
    """(role, barrier, phase) of every wait that can find its barrier two phases on; fails when a role does not reach its end."""
    run = _runner(roles)
    pos, _ = run()
    assert all(pos[name] == len(role) for name, role in roles.items()), pos
    missed = []
    for name, role in roles.items():
        for at, (op, bar, phase) in enumerate(role):
            if op == "wait" and run(name, at)[1][bar] > phase + 1:
                missed.append((name, bar, phase))
    return missed


def phases_early(roles):
    """(role, barrier, phase) of every wait that can come while the phase before the one it names is still open."""
    run = _runner(roles)
    early = set()
    for held, role in roles.items():
        done = {}
        for at, (op, bar, _) in enumerate(role):
            if op != "arrive":
                continue
            open_phase = done[bar] = done.get(bar, -1) + 1  # held ahead of its arrival, this phase stays open
            pos, _ = run(held, at)
            for name, other in roles.items():
                early |= {(name, b, ph) for b, ph in ((b, ph) for o, b, ph in other[:pos[name] + 1] if o == "wait") if b == bar and ph == open_phase + 1}
    return early


def out_of_order(roles, first, second, lag=0):
    """Marks (second, k + lag) that a role can come to while another is still ahead of its mark (first, k)."""
    run, found = _runner(roles), set()
    for held, role in roles.items():
        for at, (op, what, k) in enumerate(role):
            if (op, what) == ("mark", first):
                pos, _ = run(held, at)
                found |= {(name, second, k + lag) for name, other in roles.items() if name != held and ("mark", second, k + lag) in other[:pos[name]]}
    return found


def test_one_barrier_for_two_buffers_is_missed():
    assert ("mma", "DS_FULL0") in {m[:2] for m in phases_missed(dq_tf32([4], 1))}
    assert ("dp_dq", "DS_FULL0") in {m[:2] for m in phases_missed(dq_bf16(4, 1))}


@pytest.mark.parametrize("items", [[1], [2], [1, 1, 1], [5, 2, 1, 3], [7, 6]])
def test_tf32_dq_waits_see_every_phase(items):
    with open(os.path.join(CSRC, "attn_bwd_sm100.cu")) as f:
        enum = re.search(r"namespace dq \{\s*enum Bar \{(.*?)\}", f.read(), re.S).group(1)
    ds_bars = len(re.findall(r"\bDS_FULL\d?\b", enum))
    assert phases_missed(dq_tf32(items, ds_bars)) == []
    assert phases_early(dq_tf32(items, ds_bars)) == set()


@pytest.mark.parametrize("items", [[1], [2], [1, 1, 1], [5, 2, 1, 3], [4, 3]])
def test_tf32_dkdv_waits_see_their_phase(items):
    roles = dkdv_tf32(items)
    assert phases_missed(roles) == []
    assert phases_early(roles) == set()


@pytest.mark.parametrize("n_kv", [1, 2, 3, 9])
def test_bf16_dq_waits_see_every_phase(n_kv):
    with open(os.path.join(CSRC, "attn_bwd_bf16_sm100.cu")) as f:
        enum = re.search(r"namespace dq16 \{\s*enum Bar \{(.*?)\}", f.read(), re.S).group(1)
    enum = re.sub(r"//[^\n]*", "", enum)
    at, value = {}, -1
    for name, explicit in re.findall(r"(\w+)(?:\s*=\s*(\d+))?\s*(?:,|$)", enum):
        value = int(explicit) if explicit else value + 1
        at[name] = value
    ds_bars = min(v for v in at.values() if v > at["DS_FULL"]) - at["DS_FULL"]
    assert phases_missed(dq_bf16(n_kv, ds_bars)) == []


# head dimension 64: two issuers, two S^T buffers; 128: one of each
@pytest.mark.parametrize("issuers,s_bufs", [(2, 2), (1, 1)])
@pytest.mark.parametrize("n_it", [1, 2, 3, 5, 11])
def test_bf16_dkdv_waits_see_their_phase_and_statistics_stay_until_used(n_it, issuers, s_bufs):
    with open(os.path.join(CSRC, "attn_bwd_bf16_sm100.cu")) as f:
        text = f.read()
    assert re.search(r"kIssuers = HD_ == 64 \? 2 : 1;", text) and re.search(r"kSBufs = HD_ == 64 \? 2 : 1;", text)
    roles = dkdv_bf16(n_it, issuers, s_bufs)
    assert phases_missed(roles) == []
    assert phases_early(roles) == set()
    for stat, places in (("lse", s_bufs), ("delta", 1)):
        assert out_of_order(roles, stat + " staged", stat + " used") == set()
        assert out_of_order(roles, stat + " used", stat + " staged", places) == set()
    if n_it > s_bufs > 1:  # one place would not do
        assert out_of_order(roles, "lse used", "lse staged", 1) != set()


# passes (FORWARD, DV, DQ, DK) by the head sizes' buffers of the second streamed tile
@pytest.mark.parametrize("two,keys,st2", [(False, False, 2), (False, True, 2), (True, False, 2), (True, True, 2), (True, False, 1), (True, True, 1)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 9])
def test_split_waits_see_their_phase_and_statistics_stay_until_read(n, two, keys, st2):
    with open(os.path.join(CSRC, "attn_split_sm100.cu")) as f:
        text = f.read()
    assert "ST1 = 2, ST2 = TWO && SLABS == 2 ? 1 : 2;" in text and "sStats + (j % 3) * C::NSTATS * BN" in text
    roles = split(n, two, keys, st2)
    assert phases_missed(roles) == []
    assert phases_early(roles) == set()
    if keys:
        assert out_of_order(roles, "stats written", "stats read") == set()
        assert out_of_order(roles, "stats read", "stats written", 3) == set()
        if n > 1:
            assert out_of_order(roles, "stats read", "stats written", 1) != set()  # one buffer would not do
