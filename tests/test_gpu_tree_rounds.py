"""The parent rounds where they pass from the whole GPU to the cluster of blocks and on to
the single block (65,536 and 512 nodes a level), and the sort's passes: every field of the
tree bit for bit against the oracle."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu

FIELDS = ["cx", "cy", "hw", "mass", "comx", "comy", "body_start", "body_end", "parent", "is_leaf", "child",
          "level_start"]
BOX = (0.0, 100.0, 0.0, 100.0)


def _bodies(kind, n):
    b = presets.uniform(n, seed=n)
    if kind == "one cell":  # every key alike: one segment a level, grouped by fours
        b.x[:], b.y[:] = 50.0, 50.0
    elif kind == "clusters":  # a few dense cells and a sparse rest: segments longer than a thread's run
        b.x[: n // 2] = 10.0 + 1e-4 * (b.x[: n // 2] - 50.0)
        b.y[: n // 2] = 20.0 + 1e-4 * (b.y[: n // 2] - 50.0)
    elif kind == "column":  # the x digits are uniform: passes that copy
        b.x[:] = 3.0
    return b


@pytest.mark.parametrize("kind", ["spread", "one cell", "clusters", "column"])
@pytest.mark.parametrize("n,n_max", [(2, 1), (511, 1), (513, 1), (5_000, 1), (40_000, 2), (66_001, 1), (70_000, 1)])
def test_rounds_bit_exact(G, oracle, kind, n, n_max):
    b = _bodies(kind, n)
    ob = oracle.Bodies.from_arrays(b.x, b.y, b.mass, b.vx, b.vy)
    t = oracle.tree_build(ob, n_max, BOX)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4))
    for _ in range(2):  # the second build starts from the first one's sizes
        gb = b.copy()
        ctx.build_tree(gb, n_max, BOX)
        d = ctx.export_tree()
        assert d.n_nodes == t.n_nodes and d.n_levels == t.n_levels
        for f in FIELDS:
            assert np.array_equal(getattr(d, f), getattr(t, f), equal_nan=True), f
        assert np.array_equal(gb.x, ob.x) and np.array_equal(gb.y, ob.y) and np.array_equal(gb.mass, ob.mass)
