"""Parent rounds past the 31st, whose shift the reference takes modulo 64 (a masked shift): the
levels of a tree whose bodies lie in an order without runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOX = (0.0, 100.0, 0.0, 100.0)


def _level_sizes(keys):
    """Node counts of the rounds of Tree::build over one-body leaves with these keys."""
    first, shift, sizes = np.arange(len(keys)), 2, [len(keys)]
    while len(first) > 1:
        g = keys[first] >> np.uint64(shift & 63)
        head = np.r_[True, g[1:] != g[:-1]]
        i = np.arange(len(first))
        start = np.maximum.accumulate(np.where(head, i, 0))
        first = first[(i - start) % 4 == 0]
        sizes.append(len(first))
        shift += 2
    return sizes


def test_rounds_past_the_key(G):
    """Neighbours on both sides of the box's middle line, one after the other: no two in a row
    share a cell below the root, so nothing is grouped before the shift has left the key behind
    (20 rounds), and 4^11 + 2 leaves are two nodes when it starts again from 0.  They stay apart
    until it has passed the bit in which they differ once more."""
    n = 4 ** 11 + 2
    k = np.arange(n)
    b = G.Bodies.from_arrays((k // 2 + 0.5) * (200.0 / n), 50.0 + np.where(k % 2 == 0, -1e-3, 1e-3), np.ones(n))
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0))
    sizes = _level_sizes(ctx.morton_encode(b.x, b.y, BOX))
    assert sizes[20] == n and sizes[31:53] == [2] * 22 and sizes[53:] == [1]
    ctx.build_tree(b, 1, BOX, balanced=True)
    nn, nl, lv, _ = ctx.tree_info()
    ctx.close()
    assert (nl, lv, nn) == (n, len(sizes), sum(sizes))
