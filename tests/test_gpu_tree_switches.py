"""The parent rounds at the sizes where their kernels change: one block or a cluster (4,096
leaves), fields by the whole GPU or by one cluster (2,048 nodes a level), rounds by the whole GPU or
by one cluster (65,536 nodes a level); every field of the tree bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_tree_rounds import BOX, FIELDS, _bodies

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spread", "one cell", "clusters"])
@pytest.mark.parametrize("n", [2_047, 2_048, 2_049, 4_095, 4_096, 4_097, 65_535, 65_536, 65_537])
def test_rounds_at_the_switches(G, oracle, kind, n):
    b = _bodies(kind, n)
    ob = oracle.Bodies.from_arrays(b.x, b.y, b.mass, b.vx, b.vy)
    t = oracle.tree_build(ob, 1, BOX)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4))
    for _ in range(2):  # the second build starts from the first one's sizes
        gb = b.copy()
        ctx.build_tree(gb, 1, BOX)
        d = ctx.export_tree()
        assert d.n_nodes == t.n_nodes and d.n_levels == t.n_levels
        for f in FIELDS:
            assert np.array_equal(getattr(d, f), getattr(t, f), equal_nan=True), f
        assert np.array_equal(gb.x, ob.x) and np.array_equal(gb.y, ob.y) and np.array_equal(gb.mass, ob.mass)
