"""Block trees of clusters with thousands of nodes, whose subtrees are built by
several host threads, against the oracle's recursion and (symmetric trees)
against the rule written out here: the same tasks in the same order."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G


@pytest.mark.parametrize("nt,ns,eta", [(24000, 24000, 10.0), (30000, 18000, 1.0), (24000, 300, 3.0)])
def test_tasks_match_oracle(port, nt, ns, eta):
    xt, xs = G.sphere(nt, seed=3), G.cube_surface(ns, seed=4)
    t, s = H.Cluster().build(nt, xt), H.Cluster().build(ns, xs)
    if ns > 10000:
        assert t.get_nodes()[0].shape[0] + s.get_nodes()[0].shape[0] >= 4096  # the threaded path
    assert np.array_equal(H.block_tasks(t, s, eta), port.block_tasks(port.cluster(xt), port.cluster(xs), eta))


@pytest.mark.parametrize("world", [1, 3])
def test_rank_tasks_match_oracle(port, world):
    n = 24000
    x = G.sphere(n, seed=5)
    t = H.Cluster().build(n, x, size_world=world)
    o = port.cluster(x, size_world=world)
    for r in range(world):
        assert np.array_equal(H.block_tasks_rank(t, t, 10.0, r), port.block_tasks_rank(o, o, 10.0, r))


def sym_tasks(c, eta, uplo):
    ni, nd = c.get_nodes()  # pre-order: depth, rank, offset, size, sons, counter; radius, centre
    ni, nd = ni.tolist(), nd.tolist()
    kids, stack = [[] for _ in ni], []
    for k, v in enumerate(ni):
        while stack and ni[stack[-1]][0] >= v[0]:
            stack.pop()
        if stack:
            kids[stack[-1]].append(k)
        stack.append(k)

    def adm(t, s):
        a, b = nd[t], nd[s]
        d = (a[1] - b[1], a[2] - b[2], a[3] - b[3])
        dist = float(np.sqrt(abs(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])))
        return 2 * min(a[0], b[0]) < eta * max(dist - a[0] - b[0], 0.0)

    def ok(t, s):
        (to, tm), (so, sm) = ni[t][2:4], ni[s][2:4]
        if ni[t][1] < 0:
            return False
        return tm == sm if to == so else (so - to >= tm if to < so else to - so >= sm)

    out = []

    def visit(t, s, a):
        if a and ok(t, s):
            out.append((t, s, 1))
            return False
        if not kids[t] and not kids[s]:
            return True
        ks = [(p, q) for q in (kids[s] or [s]) for p in (kids[t] or [t])]
        ka = [adm(*k) for k in ks]
        quiet = [visit(p, q, b) for (p, q), b in zip(ks, ka)]
        if ni[t][3] * ni[s][3] <= 1000000 and all(quiet) and ok(t, s):
            return True
        out.extend((p, q, int(b)) for (p, q), b, z in zip(ks, ka, quiet) if z)
        return False

    if visit(0, 0, adm(0, 0)):
        out.append((0, 0, int(adm(0, 0))))
    rows = [(ni[t][2], ni[t][3], ni[s][2], ni[s][3], a) for t, s, a in out if ni[t][1] == 0]
    rows = [r for r in rows if uplo == "N" or (r[2] <= r[0] if uplo == "L" else r[2] >= r[0])]
    return np.array(sorted(rows, key=lambda r: (r[0], r[2])), np.int32)


@pytest.mark.parametrize("uplo", ["N", "L", "U"])
def test_symmetric_tasks_match_recursion(uplo):
    n = 24000
    c = H.Cluster().build(n, G.sphere(n, seed=6))
    assert 2 * c.get_nodes()[0].shape[0] >= 4096
    assert np.array_equal(H.block_tasks(c, c, 10.0, uplo, True), sym_tasks(c, 10.0, uplo))
