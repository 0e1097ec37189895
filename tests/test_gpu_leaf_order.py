"""Uploaded trees whose leaves lie in another order than their bodies, with and without a body
that is in no leaf."""
from types import SimpleNamespace

import numpy as np
import pytest

from helpers import rel_vec_err
from test_gpu_orphan_leaf import PER, _tree

pytestmark = pytest.mark.gpu


def _turned(t, nl):
    """The tree with its leaves' ids in reverse."""
    new = np.arange(t.n_nodes)
    new[:nl] = new[:nl][::-1]
    f = {k: getattr(t, k)[new] for k in ("cx", "cy", "hw", "mass", "comx", "comy", "body_start", "body_end", "is_leaf",
                                         "parent", "child")}
    f["child"] = np.where(f["child"] >= 0, new[f["child"]], -1).astype(np.int32)
    return SimpleNamespace(n_nodes=t.n_nodes, **f)


@pytest.mark.parametrize("missing", [False, True])
@pytest.mark.parametrize("turned", [False, True])
def test_leaf_order(G, turned, missing):
    """Every body's force as in body order (sums in another order: 1e-12), and a body in no leaf
    keeps a = 0 (what the others feel of its mass is the tree's business)."""
    nl = 300
    rng = np.random.default_rng(nl)
    n, gone = PER * nl, PER * 100  # the first body of a leaf in the middle
    x, y, m = np.arange(n) // PER + rng.uniform(0, 0.5, n), rng.uniform(0, 0.5, n), np.ones(n)
    got = []
    for turn in (False, turned):
        t = _tree(x, y, nl, 0)
        if missing:
            t.body_start[gone // PER] += 1
        if turn:
            t = _turned(t, nl)
        lists = SimpleNamespace(data=np.zeros((t.n_nodes, G.LIST_CAP), np.uint32), lengths=np.zeros(t.n_nodes, np.uint8))
        ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4, eps64=0.05))
        ctx.set_mode(G.MODE_ACCURATE, G.PREC_FP64, 0.5)
        ctx.upload_tree_data(t, lists, lists)
        ax, ay = np.full(n, 7.0), np.full(n, 7.0)
        for _ in range(2):
            ctx.compute_forces(x, y, m, ax, ay)
        got.append((ax, ay))
        ctx.close()
    (ax, ay), (bx, by) = got
    keep = np.arange(n) != gone if missing else np.full(n, True)
    assert rel_vec_err(bx[keep], by[keep], ax[keep], ay[keep]).max() < 1e-12
    assert (np.hypot(bx, by)[keep] > 0).all() and not bx[~keep].any() and not by[~keep].any()
