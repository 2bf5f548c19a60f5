"""The barrier protocol of fla_chunk_kernel (csrc/fla_kernel.cuh, attention mode) as an ordering problem,
on the CPU. Every role's waits and arrivals are listed in program order; an arrival by tcgen05.commit
is asynchronous, but follows the issuer's earlier ones. Three things must hold in the partial order that
follows, however long any warp is held up between two of its instructions:

* no cycle (no deadlock);
* a wait for phase n of a barrier is never overtaken by the completion of phase n + 1 (the wait tests a
  parity, and would then block for good): some arrival of phase n + 1 comes after every wait for phase n;
* every asynchronous arrival has happened before the CTA ends.
"""
import collections

import pytest


class Model:
    def __init__(self):
        self.succ = collections.defaultdict(set)
        self.nodes = 0
        self.last, self.last_async = {}, {}   # per role
        self.waits = []                       # (barrier, phase, node)
        self.arrivals = collections.defaultdict(lambda: collections.defaultdict(list))  # barrier -> role -> nodes
        self.asyncs = []

    def _node(self, role):
        n, self.nodes = self.nodes, self.nodes + 1
        if role in self.last:
            self.succ[self.last[role]].add(n)
        self.last[role] = n
        return n

    def wait(self, role, bar, phase):
        self.waits.append((bar, phase, self._node(role)))

    def arrive(self, role, bar):
        self.arrivals[bar][role].append(self._node(role))

    def commit(self, role, bar, count=1):
        issue = self._node(role)
        n, self.nodes = self.nodes, self.nodes + 1
        self.succ[issue].add(n)
        if role in self.last_async:
            self.succ[self.last_async[role]].add(n)
        self.last_async[role] = n
        self.asyncs.append((bar, n))
        self.arrivals[bar][role + "/async"].extend([n] * count)

    def faults(self, per_phase, end):
        """per_phase: barrier -> {role: arrivals of that role in one phase}."""
        def of_phase(bar, phase):
            nodes = []
            for role, count in per_phase(bar).items():
                got = self.arrivals[bar].get(role, [])[phase * count:(phase + 1) * count]
                if len(got) < count:
                    return None  # the phase does not complete in this run
                nodes += got
            return nodes

        for bar, phase, node in self.waits:
            done = of_phase(bar, phase)
            assert done is not None, f"{bar} phase {phase} is waited for and never completes"
            for n in done:
                self.succ[n].add(node)
        # topological order, then reachability as bit sets
        indeg = collections.Counter(m for s in self.succ.values() for m in s)
        order = [n for n in range(self.nodes) if indeg[n] == 0]
        for n in order:
            for m in self.succ[n]:
                indeg[m] -= 1
                if indeg[m] == 0:
                    order.append(m)
        if len(order) < self.nodes:
            return ["deadlock"]
        reach = [0] * self.nodes
        for n in reversed(order):
            for m in self.succ[n]:
                reach[n] |= reach[m] | (1 << m)
        found = []
        for bar, phase, node in self.waits:
            nxt = of_phase(bar, phase + 1)
            if nxt is not None and not any(reach[node] >> n & 1 for n in nxt):
                found.append(f"overtaken: {bar.split('@')[0]}")
        found += [f"outlives the CTA: {bar.split('@')[0]}" for bar, n in self.asyncs if not reach[n] >> end & 1]
        return sorted(set(found))


def chunk_kernel(n_iter, nslot, o_bufs, has_init, norm, to_final, split_pb=True, drain=True):
    m = Model()
    conv, epi = ["convA", "convB"], ["epi0", "epi1"]  # two warps stand for the eight and the four
    roles = ["prod0", "prod1", "X", "Y"] + conv + epi
    slot = lambda t: t % nslot  # noqa: E731
    full = lambda t: f"full@{slot(t)}"  # noqa: E731
    empty = lambda t: f"empty@{slot(t)}"  # noqa: E731
    pb = lambda i: (f"pb_ready@{i & 1}", i >> 1) if split_pb else ("pb_ready@0", i)  # noqa: E731
    o_full = lambda i: (f"o_full@{i & 1}", i >> 1)  # noqa: E731
    o_free = lambda i: (f"o_free@{i & 1}", i >> 1) if o_bufs == 2 else ("o_free@0", i)  # noqa: E731
    first = 1 if has_init else 0  # phase of sb_ready that chunk 0 completes
    for p in ("prod0", "prod1"):
        for t in range(3 * n_iter):
            if t >= nslot:
                m.wait(p, empty(t), t // nslot - 1)
            m.arrive(p, full(t))  # its bytes are counted with it; k's land on q's barrier
    def issue_qk(i):
        m.wait("X", full(3 * i), 3 * i // nslot)
        m.commit("X", "p_full@")
        m.commit("X", empty(3 * i))
        m.commit("X", empty(3 * i + 1))
    issue_qk(0)
    for i in range(n_iter):
        if i > 0 or has_init:
            m.wait("X", "sb_ready@", i - 1 + first)
        m.wait("X", full(3 * i + 2), (3 * i + 2) // nslot)
        m.commit("X", "s_full@")
        m.commit("X", empty(3 * i + 1))
        m.commit("X", empty(3 * i + 2))
        if i + 1 < n_iter:
            m.wait("X", "p_read@", i)
            if i >= 1:
                m.wait("X", *o_full(i - 1))
            issue_qk(i + 1)
    for i in range(n_iter):
        if i >= o_bufs:
            m.wait("Y", *o_free(i - o_bufs))
        if i > 0 or has_init:
            m.wait("Y", "sb_ready@", i - 1 + first)
        m.wait("Y", full(3 * i), 3 * i // nslot)
        m.commit("Y", "qs_done@")
        m.commit("Y", empty(3 * i))
        m.wait("Y", *pb(i))
        m.wait("Y", full(3 * i + 2), (3 * i + 2) // nslot)
        m.commit("Y", o_full(i)[0])
        m.commit("Y", empty(3 * i + 2))
    for c in conv:
        if has_init:
            m.arrive(c, "sb_ready@")
        for i in range(n_iter):
            m.wait(c, "p_full@", i)
            m.arrive(c, "p_read@")
            m.arrive(c, pb(i)[0])
            last = i == n_iter - 1
            if not last or to_final:
                m.wait(c, "s_full@", i)
                m.wait(c, "qs_done@", i)
                if not last:
                    m.arrive(c, "sb_ready@")
            if norm:
                if i > 0:
                    m.wait(c, "rs_free@", i - 1)
                m.arrive(c, "rs_full@")
    for e in epi:
        for i in range(n_iter):
            if norm:
                m.wait(e, full(3 * i), 3 * i // nslot)
                if i > 0:
                    m.wait(e, "vec_ready@", i - 1)
                m.arrive(e, "vec_ready@")
                m.arrive(e, empty(3 * i))
                m.arrive(e, empty(3 * i + 1))
            m.wait(e, *o_full(i))
            if norm:
                m.arrive(e, empty(3 * i + 2))
                m.wait(e, "rs_full@", i)
                m.arrive(e, "rs_free@")
            m.arrive(e, o_free(i)[0])
    if drain:
        for r in ("X", "Y"):
            m.commit(r, f"drained_{r}@")
            m.wait(r, f"drained_{r}@", 0)
    for r in roles:
        m.arrive(r, "end")
    end = m._node("sync")
    for nodes in m.arrivals["end"].values():
        m.succ[nodes[0]].add(end)

    def per_phase(bar):
        if bar.startswith("full"):
            return {"prod0": 1, "prod1": 1}
        if bar.startswith(("pb_ready", "sb_ready", "p_read", "rs_full")):
            return {c: 1 for c in conv}
        if bar.startswith(("o_free", "rs_free", "vec_ready")):
            return {e: 1 for e in epi}
        if bar.startswith("empty"):
            return {"in pass order": 2 + (len(epi) if norm else 0)}
        return {("Y" if bar.startswith(("qs_done", "o_full", "drained_Y")) else "X") + "/async": 1}

    # A slot's tile changes from pass to pass, and with it who releases it: q and v by X and Y, k by X
    # twice. Bring the arrivals into pass order.
    for s in range(nslot):
        took = collections.Counter()
        for t in range(s, 3 * n_iter, nslot):
            want = {"X/async": 2} if t % 3 == 1 else {"X/async": 1, "Y/async": 1}
            if norm:
                want.update({e: 1 for e in epi})
            for role, count in want.items():
                got = m.arrivals[f"empty@{s}"][role][took[role]:took[role] + count]
                m.arrivals[f"empty@{s}"]["in pass order"] += got
                took[role] += count
    return m.faults(per_phase, end)


SHAPES = [(n, *ring, init, norm, final)
          for n in (1, 2, 3, 7) for ring in ((5, 1), (9, 2))
          for init, norm, final in ((0, 0, 0), (1, 0, 0), (0, 0, 1), (1, 0, 1), (0, 1, 0), (0, 1, 1))]


@pytest.mark.parametrize("n_iter,nslot,o_bufs,has_init,norm,to_final", SHAPES)
def test_no_wait_is_overtaken_and_nothing_outlives_the_cta(n_iter, nslot, o_bufs, has_init, norm, to_final):
    assert chunk_kernel(n_iter, nslot, o_bufs, has_init, norm, to_final) == []


def test_the_model_sees_both_mistakes():
    """One pb_ready barrier for all chunks; no wait for what the issuers issued last."""
    assert "overtaken: pb_ready" in chunk_kernel(4, 9, 2, 0, 0, 0, split_pb=False)
    assert "overtaken: pb_ready" in chunk_kernel(4, 5, 1, 1, 0, 0, split_pb=False)
    assert "outlives the CTA: s_full" in chunk_kernel(4, 5, 1, 0, 0, 0, drain=False)
    assert "outlives the CTA: empty" in chunk_kernel(4, 9, 2, 0, 0, 1, drain=False)
