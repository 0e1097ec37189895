"""The upward pass where its launches change: single-child levels apart or in the cluster
kernel, levels around its 512 nodes, rows that are not finite."""
import numpy as np
import pytest

from galax_gb300 import presets
from helpers import oracle_case, rel_vec_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_max,p", [(2, 1, 4), (40, 1, 3), (511 * 4, 4, 4), (513 * 4, 4, 4), (8_200, 8, 2),
                                       (20_000, 32, 4), (30_000, 9, 5), (3_000, 8, 8)])
def test_ref_upward_levels(G, oracle, n, n_max, p):
    """REF forces against the oracle (1e-10 per body), and the same bits when repeated."""
    b = presets.uniform(n, seed=n)
    bounds = presets.BOUNDS["uniform"]
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, bounds, p)
    ref = ob.copy()
    oracle.compute_fmm_force(ref, t, v, u, p, eps, oracle.MODE_REF)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p))
    ctx.set_params(p, eps)
    ctx.build_tree(b, n_max, bounds)
    out = []
    for _ in range(2):
        ax, ay = np.zeros(n), np.zeros(n)
        ctx.compute_forces(b.x, b.y, b.mass, ax, ay)
        out.append((ax, ay))
    assert (rel_vec_err(*out[0], ref.ax, ref.ay) <= 1e-10).all()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_non_finite_moments_are_zeroed_once(G, oracle):
    """Moments that overflow are zeroed after the pass, as in the oracle; the next evaluation
    of the same context, with masses that do not overflow, is clean."""
    n, n_max, p = 3_000, 16, 4
    b = presets.uniform(n, seed=8)
    bounds = presets.BOUNDS["uniform"]
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, bounds, p)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p))
    ctx.set_params(p, eps)
    ctx.build_tree(b, n_max, bounds)
    ax, ay = np.zeros(n), np.zeros(n)
    for scale in (1.0, 1e305, 1.0):
        ref = ob.copy()
        ref.mass[:] = ob.mass * scale
        with np.errstate(all="ignore"):
            oracle.compute_fmm_force(ref, t, v, u, p, eps, oracle.MODE_REF)
            ctx.compute_forces(b.x, b.y, np.ascontiguousarray(ref.mass), ax, ay)
            if scale == 1.0:
                assert (rel_vec_err(ax, ay, ref.ax, ref.ay) <= 1e-10).all()


def test_uploaded_tree_that_leaves_a_body_out(G, oracle):
    """A body in no leaf keeps a = 0 and is still sanitised; the others are those of the tree."""
    n, n_max, p = 400, 16, 4
    b = presets.uniform(n, seed=12)
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, presets.BOUNDS["uniform"], p)
    t.body_start[t.body_start == 0] = 1
    ob.mass[0] = -1.0
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p))
    ctx.set_params(p, eps)
    ctx.upload_tree_data(t, v, u)
    ax, ay = np.full(n, 7.0), np.full(n, 7.0)
    for _ in range(2):
        ctx.compute_forces(ob.x, ob.y, ob.mass, ax, ay)
        assert ax[0] == 0.0 and ay[0] == 0.0 and np.isfinite(ax).all() and np.abs(ax[1:]).min() > 0.0
        assert ctx.last_status() == G.STATUS_SANITIZED
    out = G.Bodies.new(n)
    ctx.download_bodies(out)
    assert out.mass[0] == 1.0
