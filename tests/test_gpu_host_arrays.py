"""Host arrays read and written by kernels, by copies or page-locked, give the same bits: sizes
on both sides of a page, of the page limit and of the kernel copy's limit, odd addresses."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu
NAMES = ("x", "y", "vx", "vy", "mass", "ax", "ay")


@pytest.mark.parametrize("n", [1, 511, 513, 8_193, 65_537, 262_145])
@pytest.mark.parametrize("offset", [0, 1])
def test_round_trips(G, n, offset):
    rng = np.random.default_rng(n)
    arrs = [rng.standard_normal(n + offset)[offset:] for _ in NAMES]
    b = G.Bodies(*arrs)
    before = [a.copy() for a in arrs]
    ctx = G.GpuContext(G.GpuConfig(max_n=n))
    ctx.upload_bodies(b)
    out = G.Bodies(*[np.full(n + offset, np.nan)[offset:] for _ in NAMES])
    ctx.download_bodies(out)
    for name, a in zip(NAMES, before):
        assert np.array_equal(getattr(out, name), a) and np.array_equal(getattr(b, name), a), name
    pinned = [G.HostArray(n) for _ in NAMES]
    ctx.download_bodies(G.Bodies(*[h.array for h in pinned]))
    for h, a in zip(pinned, before):
        assert np.array_equal(h.array, a)
    assert np.array_equal(ctx.body_ids(), np.arange(n))


@pytest.mark.parametrize("n", [700, 70_001])
def test_forces_and_permutation(G, n):
    b = presets.uniform(n, seed=n)
    bounds = presets.BOUNDS["uniform"]
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=3))
    ctx.upload_bodies(b)
    perm = ctx.rebuild_resident(16, bounds, want_perm=True)
    ids = ctx.body_ids()
    assert np.array_equal(np.sort(perm), np.arange(n)) and np.array_equal(perm, ids)
    s = G.Bodies.new(n)
    ctx.download_bodies(s)
    assert np.array_equal(s.x, b.x[perm]) and np.array_equal(s.mass, b.mass[perm])
    ax, ay = np.zeros(n), np.zeros(n)
    got = []
    for _ in range(3):  # the first evaluation makes the plan after a copy, the others read in place
        ctx.compute_forces(s.x, s.y, s.mass, ax, ay)
        got.append((ax.copy(), ay.copy()))
    host = [G.HostArray(n) for _ in range(5)]
    for h, a in zip(host, (s.x, s.y, s.mass)):
        h.array[:] = a
    ctx.compute_forces(*[h.array for h in host])
    got.append((host[3].array.copy(), host[4].array.copy()))
    out = G.Bodies.new(n)
    ctx.download_bodies(out)
    got.append((out.ax, out.ay))
    for g in got[1:]:
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1])
