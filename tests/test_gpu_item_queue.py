"""Evaluations whose items and units are taken from a queue (58,368 and more of a kind): every
item once, whatever block takes it."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,n,n_max,p,prec", [
    ("uniform", 1_000_003, 32, 4, "MIXED"),   # P2P with body masks, M2P and P2L in pairs
    ("uniform", 1_000_003, 32, 6, "MIXED"),   # M2P a lane a body, P2L as a stream
    ("disk", 1_000_003, 16, 4, "MIXED"),      # leaves of half a row
    ("uniform", 1_500_001, 48, 5, "MIXED"),   # leaves of two rows
    ("uniform", 1_000_003, 32, 4, "FP64"),
])
def test_queued_items_are_all_done_once(G, preset, n, n_max, p, prec):
    """Forces of 400 bodies against the direct sum within 16 theta^(p+1) of the rms force (a
    far pair's truncation is theta^(p+1) of its force; the sizes of a body's far forces sum to
    several times their vector sum), and the same bits when repeated: the counters are back at
    0.  A missed or doubled item of 32 leaves changes its bodies' forces by whole fractions."""
    theta = 0.35
    b = presets.make(preset, n, seed=31)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=1 << 22, p=p, eps64=0.05))
    ctx.build_tree(b, n_max, presets.BOUNDS[preset])
    ctx.set_mode(G.MODE_ACCURATE, getattr(G, "PREC_" + prec), theta)
    ctx.upload_bodies(b)
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
    err = np.hypot(got[0][0][idx] - ex, got[0][1][idx] - ey) / rms
    assert err.max() <= 16 * theta ** (p + 1), err.max()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
