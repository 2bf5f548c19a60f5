"""The barrier protocol of fla_backward_kernel (csrc/fla_backward.cuh) as an ordering problem, on the CPU:
the same three properties as in test_barrier_protocol.py, and that no buffer that several roles use in turn
(tile slots, states, their operand copies, score tiles, accumulators, the 128-wide stage) is touched out of order.
And the same for fla_taylor_attention_kernel (csrc/fla_taylor_attention.cuh) in its three roles."""
import collections

import pytest
from test_barrier_protocol import Model


class Buffers(Model):
    """Also records which nodes touch a buffer, and the order the kernel means them to have."""

    def __init__(self):
        super().__init__()
        self.uses = collections.defaultdict(list)  # buffer -> [(key, node)], key in intended order

    def touch(self, role, buf, key):
        self.uses[buf].append((key, self._node(role)))

    def mma(self, role, reads):
        """An asynchronous use: it lies between its issue and the issuer's next commit."""
        for buf, key in reads:
            issue = self._node(role)
            n, self.nodes = self.nodes, self.nodes + 1
            self.succ[issue].add(n)
            if role in self.last_async:
                self.succ[self.last_async[role]].add(n)
            self.last_async[role] = n
            self.uses[buf].append((key, n))

    def disorder(self):
        indeg = collections.Counter(m for s in self.succ.values() for m in s)
        order = [n for n in range(self.nodes) if indeg[n] == 0]
        for n in order:
            for m in self.succ[n]:
                indeg[m] -= 1
                if indeg[m] == 0:
                    order.append(m)
        reach = [0] * self.nodes
        for n in reversed(order):
            for m in self.succ[n]:
                reach[n] |= reach[m] | (1 << m)
        bad = []
        for buf, uses in self.uses.items():
            groups = collections.defaultdict(list)
            for key, n in uses:
                groups[key].append(n)
            keys = sorted(groups)
            for a, b in zip(keys, keys[1:]):
                bad += [buf for m in groups[a] for n in groups[b] if not reach[m] >> n & 1]
        return sorted(set(bad))


def backward_kernel(n_iter, double, has_r, to_final, wait_dv=True, early_release=False):
    m = Buffers()
    conv, state, epi = ["convA", "convB"], ["stateA", "stateB"], ["epi0", "epi1"]  # two warps stand for each group
    roles = ["prod0", "prod1", "X"] + conv + state + epi
    nslot = 8 if double else 4
    V, G, K, Q = range(4)

    def slot(i, w):  # slot and how often it was filled before, as slot_of() and use_of()
        if double:
            return (4 * i + w) % nslot, (4 * i + w) // nslot
        return (w - i) & 3, i

    tiles = [slot(i, w) for i in range(n_iter) for w in range(4)]
    for p in ("prod0", "prod1"):
        for s, use in tiles:
            if use > 0:
                m.wait(p, f"empty@{s}", use - 1)
            m.touch(p, f"tile{s}", (use, 0))
            m.arrive(p, f"full@{s}")
    X = "X"
    m.wait(X, "s_loaded@", 0)
    alt = lambda name, n: (f"{name}@{n & 1}", n >> 1)  # noqa: E731
    place = lambda n: n & 1 if double else 0  # noqa: E731
    tile = lambda i, w: m.wait(X, f"full@{slot(i, w)[0]}", slot(i, w)[1])  # noqa: E731
    release = lambda i, w: m.commit(X, f"empty@{slot(i, w)[0]}")  # noqa: E731
    reads = lambda i, *ws: [(f"tile{slot(i, w)[0]}", (slot(i, w)[1], 1)) for w in ws]  # noqa: E731

    def scores(n):
        i, which = divmod(n, 3)
        for t in ((V, G), (K, Q), ())[which]:
            tile(i, t)
        m.mma(X, [(f"P{place(n)}", (n, 0))] + reads(i, *((V, G), (K, Q), (G, V))[which]))
        m.commit(X, alt("p_full", n)[0])
        if which == 2:
            release(i, V)

    def state_term(n, copy):
        before = n - (2 if double else 1)
        if before >= 0:
            m.wait(X, *alt("o_free", before))
        if copy:
            m.mma(X, [copy, (f"O{place(n)}", (n, 0))] + reads(n // 3, (V, K, G)[n % 3]))

    def finish(n):
        m.mma(X, [(f"P{place(n)}", (n, 2)), (f"O{place(n)}", (n, 0))] + reads(n // 3, (Q, G, K)[n % 3]))
        m.commit(X, alt("o_full", n)[0])

    if double:
        scores(0)
    for i in range(n_iter):
        n = 3 * i
        have_r, want_r = i > 0 or has_r, i + 1 < n_iter or to_final
        scores(n + 1 if double else n)
        tile(i, K)
        m.mma(X, [("S", (i, 0))] + reads(i, K, V))
        m.commit(X, "s_full@")
        if i > 0:
            m.wait(X, "rb_ready@", i - 1)
        elif has_r:
            m.wait(X, "r_loaded@", 0)
        state_term(n, have_r and ("Rb", (i, 1)))
        m.wait(X, *alt("pb_ready", n))
        tile(i, Q)
        finish(n)
        scores(n + 2 if double else n + 1)
        if want_r:
            m.mma(X, [("R", (i, 0))] + reads(i, Q, G))
            m.commit(X, "r_full@")
        release(i, Q)
        state_term(n + 1, have_r and ("Rb", (i, 1)))
        m.wait(X, *alt("pb_ready", n + 1))
        finish(n + 1)
        if not double:
            scores(n + 2)
        elif i + 1 < n_iter:
            scores(n + 3)
        m.wait(X, "sb_ready@", i)
        state_term(n + 2, ("Sb", (i, 3)))
        release(i, G)
        m.wait(X, *alt("pb_ready", n + 2))
        if early_release:
            release(i, K)
        finish(n + 2)
        if not early_release:
            release(i, K)
    m.commit(X, "drained@")
    m.wait(X, "drained@", 0)
    for c in conv:
        m.touch(c, "stage", -1)  # transposes of the states at the start
        m.touch(c, "S", (-1, 0))
        m.arrive(c, "s_loaded@")
        if has_r:
            m.touch(c, "stage", -1)
            m.touch(c, "Rb", (0, 0))
            m.touch(c, "R", (-1, 0))
            m.arrive(c, "r_loaded@")
        for n in range(3 * n_iter):
            m.wait(c, *alt("p_full", n))
            m.touch(c, f"P{place(n)}", (n, 1))
            m.arrive(c, alt("pb_ready", n)[0])
    for c in state:
        for i in range(n_iter):
            last = i + 1 == n_iter
            m.wait(c, "s_full@", i)
            m.touch(c, "S", (i, 1))
            m.touch(c, "Sb", (i, 2))
            m.arrive(c, "sb_ready@")
            if not last or to_final:
                if wait_dv:
                    m.wait(c, *alt("o_full", 3 * i + 1))
                m.wait(c, "r_full@", i)
                m.touch(c, "R", (i, 1))
                m.touch(c, "Rb", (i + 1, 0))
                if not last:
                    m.arrive(c, "rb_ready@")
    for e in epi:
        for n in range(3 * n_iter):
            m.wait(e, *alt("o_full", n))
            m.touch(e, f"O{place(n)}", (n, 1))
            if e == "epi0":  # (every warp has its own rows of the stage)
                m.touch(e, "stage", n)
            m.arrive(e, alt("o_free", n)[0])
    for r in roles:
        m.arrive(r, "end")
    end = m._node("sync")
    for nodes in m.arrivals["end"].values():
        m.succ[nodes[0]].add(end)

    def per_phase(bar):
        if bar.startswith("full"):
            return {"prod0": 1, "prod1": 1}
        if bar.startswith(("pb_ready", "s_loaded", "r_loaded")):
            return {c: 1 for c in conv}
        if bar.startswith(("sb_ready", "rb_ready")):
            return {c: 1 for c in state}
        if bar.startswith("o_free"):
            return {e: 1 for e in epi}
        return {"X/async": 1}

    found = m.faults(per_phase, end)
    return found if found == ["deadlock"] else found + [f"disorder: {b}" for b in m.disorder()]


@pytest.mark.parametrize("n_iter", [1, 2, 3, 7])
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("has_r,to_final", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_no_wait_is_overtaken_and_every_shared_buffer_has_one_user(n_iter, double, has_r, to_final):
    assert backward_kernel(n_iter, double, has_r, to_final) == []


def test_the_model_sees_a_copy_overwritten_under_a_product():
    assert "disorder: Rb" in backward_kernel(3, False, 0, 0, wait_dv=False)
    assert "disorder: Rb" in backward_kernel(3, True, 1, 0, wait_dv=False)


@pytest.mark.parametrize("double", [False, True])
def test_the_model_sees_a_tile_released_before_its_last_reader(double):
    assert any(f.startswith("disorder: tile") for f in backward_kernel(7, double, 0, 0, early_release=True))


def taylor_kernel(n_iter, want_o, want_dx, early_z=False, wait_dx=True, wait_free=True):
    m = Buffers()
    conv, outs, gens = ["conv0", "conv1"], ["out0", "out1"], ["gen0", "gen1"]  # two warps stand for each group
    X, roles = "X", ["prod", "X"] + conv + outs + gens
    full, empty = lambda i: f"full@{i & 1}", lambda i: f"empty@{i & 1}"  # noqa: E731
    for i in range(n_iter):
        if i >= 2:
            m.wait("prod", empty(i), (i >> 1) - 1)
        m.touch("prod", f"ab{i & 1}", (i, 0))
        m.arrive("prod", full(i))
    for i in range(n_iter):
        last, have_z = i + 1 == n_iter, i > 0
        ab, raw = (f"ab{i & 1}", (i, 1)), f"raw{i & 1}"
        m.wait(X, "y_ready@", i)
        m.wait(X, full(i), i >> 1)
        if want_dx and have_z and wait_dx:
            m.wait(X, "dx_free@", i - 1)
        m.mma(X, [(raw, (i, 1)), ("P", (i, 0))])
        if want_dx:
            m.mma(X, [ab, ("T", (i, 0))])
        m.commit(X, "p_full@")
        if have_z:
            m.wait(X, "zb_ready@", i - 1)
        if not last:
            m.mma(X, [ab, ("y", (i, 1)), ("Z", (i, 0))])
            m.commit(X, "y_free@")
        if want_o:
            m.wait(X, "x_ready@", i)
            if have_z:
                m.wait(X, "o_free@", i - 1)
                m.mma(X, [("x", (i, 1)), ("Zb", (i, 1)), ("O", (i, 0))])
            if not last:
                m.commit(X, "x_free@")
        if not last and (early_z or not want_dx):
            m.commit(X, "z_full@")
        m.wait(X, "pb_ready@", i)
        if want_o:
            m.mma(X, [ab, ("P", (i, 2)), ("O", (i, 0))])
            m.commit(X, "o_full@")
        if want_dx:
            if have_z:  # the gradient of phi(x), into the place of the scores
                m.mma(X, [ab, ("Zb", (i, 1)), ("P", (i, 3))])
            m.mma(X, [(raw, (i, 1)), ("T", (i, 2))])  # T y, into a part of T that has been read
            m.commit(X, "dx_full@")
            if not last and not early_z:
                m.commit(X, "z_full@")
        m.commit(X, empty(i))
    m.commit(X, "drained@")
    m.wait(X, "drained@", 0)
    for c in conv:
        for i in range(n_iter):
            m.wait(c, "p_full@", i)
            m.touch(c, "P", (i, 1))
            if want_dx:
                m.touch(c, "T", (i, 1))
            m.arrive(c, "pb_ready@")
            if i + 1 < n_iter:
                m.wait(c, "z_full@", i)
                m.touch(c, "Z", (i, 1))
                m.touch(c, "Zb", (i + 1, 0))
                m.arrive(c, "zb_ready@")
    for o in outs:
        for i in range(n_iter):
            if want_dx:
                m.wait(o, "dx_full@", i)
                m.touch(o, "T", (i, 3))
                if i > 0:
                    m.touch(o, "P", (i, 4))
                m.arrive(o, "dx_free@")
            if want_o:
                m.wait(o, "o_full@", i)
                m.touch(o, "O", (i, 1))
                m.arrive(o, "o_free@")
    for g in gens:
        for i in range(n_iter):
            if i > 0 and wait_free:
                m.wait(g, "y_free@", i - 1)
            m.touch(g, f"raw{i & 1}", (i, 0))
            m.touch(g, "y", (i, 0))
            m.arrive(g, "y_ready@")
            if want_o:
                if i > 0:
                    m.wait(g, "x_free@", i - 1)
                m.touch(g, "x", (i, 0))
                m.arrive(g, "x_ready@")
    for r in roles:
        m.arrive(r, "end")
    end = m._node("sync")
    for nodes in m.arrivals["end"].values():
        m.succ[nodes[0]].add(end)

    def per_phase(bar):
        for prefix, group in (("full", ["prod"]), ("pb_ready", conv), ("zb_ready", conv), ("o_free", outs), ("dx_free", outs),
                              ("y_ready", gens), ("x_ready", gens)):
            if bar.startswith(prefix):
                return {r: 1 for r in group}
        return {"X/async": 1}

    found = m.faults(per_phase, end)
    return found if found == ["deadlock"] else found + [f"disorder: {b}" for b in m.disorder()]


ROLES = {"forward": (1, 0), "dQ": (0, 1), "dK, dV": (1, 1)}  # want_o, want_dx


@pytest.mark.parametrize("n_iter", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("role", ROLES)
def test_taylor_kernel_in_every_role(n_iter, role):
    assert taylor_kernel(n_iter, *ROLES[role]) == []


def test_the_taylor_model_sees_what_is_left_out():
    assert "disorder: Zb" in taylor_kernel(3, 0, 1, early_z=True)
    assert {"disorder: P", "disorder: T"} <= set(taylor_kernel(3, 1, 1, wait_dx=False))
    assert any(f.startswith("disorder: raw") or f == "disorder: y" for f in taylor_kernel(4, 1, 0, wait_free=False))
