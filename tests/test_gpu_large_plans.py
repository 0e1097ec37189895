"""Plans on both sides of 131,072 leaves, where their scans go from one cluster to the whole GPU
and the list starts get a kernel of their own, against the oracle."""
import numpy as np
import pytest

from galax_gb300 import presets
from helpers import oracle_case, rel_vec_err
from test_gpu_near_split import _oracle_wx

pytestmark = pytest.mark.gpu
LIMIT = 131_072


@pytest.mark.parametrize("preset,n,n_max", [("uniform", 2 * LIMIT, 2), ("uniform", 2 * LIMIT + 1, 2),
                                            ("plummer", 3 * LIMIT + 4, 3)])
def test_accurate_plan(G, oracle, preset, n, n_max):
    """FP64 forces within 1e-10 of the oracle's evaluation of its own lists (one pair more or less
    is 1e-4 and above), and its pair counts."""
    p, eps, bounds = 2, 0.05, presets.BOUNDS[preset]
    b = presets.make(preset, n, seed=n)
    ob = oracle.Bodies.from_arrays(b.x, b.y, b.mass)
    t = oracle.tree_build(ob, n_max, bounds)
    assert t.n_leaves == -(-n // n_max)
    ref, far, p2p, m2p, p2l = _oracle_wx(oracle, ob, t, 0.5, 0.4, p, eps)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p, eps64=eps))
    ctx.set_mode(G.MODE_ACCURATE, G.PREC_FP64, 0.5)
    ctx.set_near_split(0.4)
    ctx.build_tree(b, n_max, bounds)
    ax, ay = np.zeros(n), np.zeros(n)
    ctx.compute_forces(b.x, b.y, b.mass, ax, ay)
    assert ctx.plan_info()[:2] == (far.off[-1], p2p.off[-1])
    assert ctx.plan_split_info() == (m2p.off[-1], p2l.off[-1])
    assert rel_vec_err(ax, ay, ref.ax, ref.ay).max() < 1e-10


def test_ref_plan(G, oracle):
    p, n, bounds = 2, 2 * LIMIT + 1, presets.BOUNDS["uniform"]
    b = presets.uniform(n, seed=1)
    ob, t, v, u, eps = oracle_case(oracle, b, 2, bounds, p)
    ref = ob.copy()
    oracle.compute_fmm_force(ref, t, v, u, p, eps, oracle.MODE_REF)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p, eps64=eps))
    ctx.build_tree(b, 2, bounds)
    ax, ay = np.zeros(n), np.zeros(n)
    ctx.compute_forces(b.x, b.y, b.mass, ax, ay)
    assert rel_vec_err(ax, ay, ref.ax, ref.ay).max() < 1e-10
