"""Moments that overflow on the way up are zeroed after the pass, as in the oracle."""
import numpy as np
import pytest

from galax_gb300 import presets
from helpers import oracle_case, rel_vec_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 4])
def test_overflowing_moments(G, oracle, p):
    """Bodies in a box much smaller than the softening, so that of all terms only a node's total
    mass can overflow: leaves hold 6e307, two of them 1.3e308, four more than FP64 does.  Their
    moments are zero then and the forces finite; left as they are they make the far field NaN.
    The evaluation before and the one after, with masses of order 1, see none of it."""
    n, n_max = 3_000, 16
    b = presets.uniform(n, seed=8)
    b.x *= 1e-5
    b.y *= 1e-5
    bounds = (0.0, 1e-3, 0.0, 1e-3)
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, bounds, p, 1000.0)
    far, near = oracle.mac_lists_build(t, oracle.node_radii(ob, t), 0.5)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p))
    ctx.set_params(p, eps)
    ctx.set_mode(G.MODE_ACCURATE, G.PREC_FP64, 0.5)
    ctx.build_tree(b, n_max, bounds)
    ax, ay = np.zeros(n), np.zeros(n)
    for scale in (1.0, 4e306, 1.0):
        ref = ob.copy()
        ref.mass[:] = ob.mass * scale
        oracle.compute_fmm_force_mac(ref, t, far, near, p, eps)
        mult = oracle.p2m(ref, t, p)
        oracle.m2m(mult, t, p)
        zeroed = np.flatnonzero(mult.reshape(t.n_nodes, -1)[:, 0] == 0.0)
        assert np.isin(far.idx[:far.off[-1]], zeroed).any() == (scale > 1.0)
        assert np.isfinite(ref.ax).all() and np.isfinite(ref.ay).all()
        ctx.compute_forces(b.x, b.y, np.ascontiguousarray(ref.mass), ax, ay)
        assert rel_vec_err(ax, ay, ref.ax, ref.ay).max() <= 1e-10, scale
