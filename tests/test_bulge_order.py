"""Order of the bulge chase (sbtrd_kernel in eig2.cu): a model of its tasks, the band
elements that each reads and writes, and the waits between them. Every two accesses of
one element, one of them a write, must be ordered by program order and waits."""
import pytest

NB = 16


class Graph:
    """Happens-before of nodes added in an order in which it is acyclic."""

    def __init__(self):
        self.before = []   # bit set of the nodes that come before each node
        self.sweep = []
        self.access = {}   # element -> [(node, writes)]

    def add(self, sweep, preds, reads, writes):
        node, bits = len(self.before), 0
        for p in preds:
            bits |= self.before[p] | (1 << p)
        self.before.append(bits)
        self.sweep.append(sweep)
        for e in writes:
            self.access.setdefault(e, []).append((node, True))
        for e in reads - writes:
            self.access.setdefault(e, []).append((node, False))
        return node

    def conflicts(self):
        bad = []
        for e, acc in self.access.items():
            for x in range(len(acc)):
                for y in range(x + 1, len(acc)):
                    (a, wa), (b, wb) = acc[x], acc[y]
                    if (wa or wb) and not (self.before[b] >> a) & 1 and not (self.before[a] >> b) & 1:
                        bad.append((e, self.sweep[a], self.sweep[b]))
        return bad


def steps(ld, s):
    return (ld - 1 - s + NB - 1) // NB


def block(r0, c0, lower=False):
    return {(r0 + i, c0 + j) for i in range(NB) for j in range(NB) if not lower or i >= j}


def build(ld, pairs, column0):
    """column0: the second half of an E task loads its first column too."""
    g = Graph()
    pub_d, pub_e = {}, {}  # (sweep, value) -> node that publishes it
    last_d, last_e = {}, {}  # pair -> last node of its D and E warp

    def at(pub, s, value):  # the first publication of at least this value
        return min((v, n) for (t, v), n in pub.items() if t == s and v >= value)[1]

    for s in range(ld - 1):
        pair, ns, nprev = s % pairs, steps(ld, s), steps(ld, s - 1) if s else 0
        first = [at(pub_e, s - 1, 1), at(pub_d, s - 1, 2)] if s else []
        if s >= pairs:
            first.append(at(pub_e, s - pairs, 2 * steps(ld, s - pairs)))
        col = {(s + 1 + i, s) for i in range(NB)}
        prev_d = g.add(s, first + ([last_d[pair]] if pair in last_d else []), col, col)
        pub_d[(s, 1)] = prev_d
        prev_e = last_e.get(pair)
        # D (s, j) and E (s, j) alternate here; D (s, j + 1) waits for E (s, j)'s reflector,
        # E (s, j) for D (s, j - 1)
        for j in range(ns):
            p = s + 1 + NB * j
            preds = [prev_d]
            if s:
                preds += [at(pub_e, s - 1, 2 * min(j + 1, nprev)), at(pub_d, s - 1, 2 * min(j + 2, nprev))]
            if j:
                preds.append(at(pub_e, s, 2 * j - 1))
            d = block(p, p, lower=True)
            prev_d = g.add(s, preds, d, d)
            pub_d[(s, 2 * (j + 1))] = prev_d
            if j + 1 < ns:
                preds = [at(pub_d, s, max(1, 2 * j))] + ([prev_e] if prev_e is not None else [])
                if s:
                    preds += [at(pub_d, s - 1, 2 * min(j + 2, nprev)), at(pub_e, s - 1, min(2 * j + 3, 2 * nprev))]
                e = block(p + NB, p)
                prev_e = g.add(s, preds, e, e)
                pub_e[(s, 2 * j + 1)] = prev_e
                rest = {(r, c) for r, c in e if c > p}
                prev_e = g.add(s, [prev_e], e if column0 else rest, rest)
            else:
                prev_e = g.add(s, [prev_e] if prev_e is not None else [], set(), set())
            pub_e[(s, 2 * (j + 1))] = prev_e
        last_d[pair], last_e[pair] = prev_d, prev_e
    return g


@pytest.mark.parametrize("ld,pairs", [(48, 4), (64, 8), (96, 4), (96, 8)])
def test_every_conflicting_access_is_ordered(ld, pairs):
    assert build(ld, pairs, column0=False).conflicts() == []


def test_model_sees_the_load_of_a_final_column():
    """The first column of an E block, loaded in the second half, meets the next sweep."""
    bad = build(64, 8, column0=True).conflicts()
    assert bad and all(abs(a - b) == 1 for _, a, b in bad)
