"""The queued branch of the near-list split's kernels: evaluations with more items or units of
every kind than a grid has blocks to give each its own (16 turns of 24 blocks an SM)."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu
QUEUED = 16 * 24 * 152  # items of a kind from which they are queued


@pytest.mark.parametrize("n,n_max,p,prec,theta_b", [
    (1_000_003, 8, 4, "MIXED", 0.35),   # packed pairs: P2P as a stream, M2P, P2L by leaf and by body
    (1_000_003, 8, 6, "MIXED", 0.35),   # M2P a lane a body, P2L as a stream
    (1_000_003, 8, 3, "FP64", 0.35),    # the same in FP64
    (2_000_003, 40, 4, "MIXED", 0.0),   # leaves of two rows: P2P and M2P by chunks, P2L in pairs
    (2_000_003, 40, 6, "MIXED", 0.0),   # and P2L a row at a time
])
def test_split_items_are_all_done_once(G, n, n_max, p, prec, theta_b):
    """Forces of 400 bodies against the direct sum within 16 theta^(p+1) of the rms force (every
    truncation is theta^(p+1) of its force), and the same bits when repeated: the counters are
    back at 0.  A missed or doubled item changes its bodies' forces by whole fractions."""
    theta = 0.35
    b = presets.make("uniform", n, seed=31)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p, eps64=0.05))
    ctx.build_tree(b, n_max, presets.BOUNDS["uniform"])
    ctx.set_mode(G.MODE_ACCURATE, getattr(G, "PREC_" + prec), theta)
    ctx.set_near_split(theta)
    ctx.set_body_split(theta_b)
    ctx.upload_bodies(b)
    _, near, _ = ctx.plan_info()
    m2p, p2l = ctx.plan_split_info()
    # at most 32 source leaves an item or unit, 96 P2P rows a body-level unit
    assert min(near, m2p, p2l) / 32 > QUEUED
    if theta_b:
        assert near / 96 > QUEUED and ctx.plan_body_split_info()[1] > near
    got = []
    for _ in range(2):
        ctx.forces_resident()
        o = G.Bodies.new(n)
        ctx.download_bodies(o)
        got.append((o.ax.copy(), o.ay.copy()))
    idx = np.random.default_rng(3).integers(0, n, 400)
    ex, ey = ctx.n2_sampled(idx)
    ctx.close()
    rms = np.sqrt(np.mean(ex ** 2 + ey ** 2))
    assert np.hypot(got[0][0][idx] - ex, got[0][1][idx] - ey).max() <= 16 * theta ** (p + 1) * rms
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
