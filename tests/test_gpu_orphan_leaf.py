"""An uploaded tree may hold a leaf that no node has as a child: its lists are empty, and the
plan's counts are those of the tree without it."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PER = 4  # bodies of a leaf


def _tree(xs, ys, nl, extra):
    """nl leaves of PER bodies under a tree of four children a node, and extra leaves apart."""
    first, level = [], [list(range(nl + extra))]
    parent, child, rng = {}, {}, {q: (PER * q, PER * q + PER) for q in level[0]}
    ids = list(range(nl))
    nn = nl + extra
    while len(ids) > 1:
        up = []
        for i in range(0, len(ids), 4):
            for c in ids[i:i + 4]:
                parent[c] = nn
            child[nn] = ids[i:i + 4]
            rng[nn] = (rng[ids[i]][0], rng[ids[i:i + 4][-1]][1])
            up.append(nn)
            nn += 1
        ids = up
    f = {k: np.zeros(nn) for k in ("cx", "cy", "hw", "mass", "comx", "comy")}
    for q in range(nn):
        a, b = rng[q]
        f["mass"][q] = b - a
        f["comx"][q], f["comy"][q] = xs[a:b].mean(), ys[a:b].mean()
        f["cx"][q], f["cy"][q] = f["comx"][q], f["comy"][q]
        f["hw"][q] = max(np.ptp(xs[a:b]), np.ptp(ys[a:b])) / 2
    ch = np.full((nn, 4), -1, np.int32)
    for q, c in child.items():
        ch[q, :len(c)] = c
    return SimpleNamespace(n_nodes=nn, child=ch, parent=np.array([parent.get(q, -1) for q in range(nn)], np.int32),
                           body_start=np.array([rng[q][0] for q in range(nn)]),
                           body_end=np.array([rng[q][1] for q in range(nn)]),
                           is_leaf=np.array([q not in child for q in range(nn)], np.uint8), **f)


@pytest.mark.parametrize("nl", [200, 1200])  # levels of one block, and of more nodes
def test_counts_with_an_orphan_leaf(G, nl):
    rng = np.random.default_rng(nl)
    n = PER * (nl + 1)
    k = np.arange(n) // PER  # leaves along a line, a little apart
    x, y, m = k + rng.uniform(0, 0.5, n), rng.uniform(0, 0.5, n), np.ones(n)
    got = []
    for extra in (0, 1):
        t = _tree(x, y, nl, extra)
        nb = PER * (nl + extra)
        lists = SimpleNamespace(data=np.zeros((t.n_nodes, G.LIST_CAP), np.uint32), lengths=np.zeros(t.n_nodes, np.uint8))
        ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4, eps64=0.05))
        ctx.set_mode(G.MODE_ACCURATE, G.PREC_FP64, 0.5)
        ctx.upload_tree_data(t, lists, lists)
        ax, ay = np.zeros(nb), np.zeros(nb)
        ctx.compute_forces(x[:nb], y[:nb], m[:nb], ax, ay)
        got.append((ctx.plan_info(), ax, ay))
        ctx.close()
    (a, ax, ay), (b, bx, by) = got
    # interactions are target bodies times source bodies less one a target, the orphan's too
    assert b == (a[0], a[1], a[2] - PER)
    assert np.array_equal(bx[:-PER], ax) and np.array_equal(by[:-PER], ay)
    assert not bx[-PER:].any() and not by[-PER:].any()
