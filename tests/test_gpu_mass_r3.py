"""m r^-3 from the integer pipes (gx_mass_r3.cuh) through the entry points that use it: the
sampled exact sum over the whole exponent range, and the FP64 near field at the leaf sizes
where its rows, half-warps and items begin and end."""
import numpy as np
import pytest

from galax_gb300 import presets
from helpers import oracle_case, rel_vec_err

pytestmark = pytest.mark.gpu


def _sum64(x, y, m, eps):
    """The plain FP64 formula and the sum of its terms' magnitudes."""
    with np.errstate(all="ignore"):
        dx, dy = x[None] - x[:, None], y[None] - y[:, None]
        r2 = dx * dx + dy * dy + eps * eps
        ir = 1.0 / np.sqrt(r2)
        f = m[None] * (ir * ir * ir)
        np.fill_diagonal(f, 0.0)
        return (f * dx).sum(1), (f * dy).sum(1), np.abs(f * dx).sum(1), np.abs(f * dy).sum(1)


@pytest.mark.parametrize("n", [2, 33, 700])
@pytest.mark.parametrize("lx,lm", [(0, 0), (60, 150), (199, 290), (205, 310), (330, 0)])
def test_sampled_sum_over_the_exponent_range(G, n, lx, lm):
    """Distances and masses over 2^-lx .. 2^lx and 2^-lm .. 2^lm, inside the integer path's
    range, across its edges and outside.  Every term has at most 8 roundings on either side,
    and a sum of n terms n more: n + 16 units of 2^-53 of the terms' magnitudes."""
    rng = np.random.default_rng(n + lx)
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(-lx, lx + 1, n)) * rng.choice([-1, 1], n)
    y = np.ldexp(rng.uniform(1, 2, n), rng.integers(-lx, lx + 1, n))
    m = np.ldexp(rng.uniform(1, 2, n), rng.integers(-lm, lm + 1, n))
    ctx = G.GpuContext(G.GpuConfig(max_n=n))
    ctx.set_params(2, 0.0)
    ctx.upload_bodies(G.Bodies.from_arrays(x, y, m))
    ax, ay = ctx.n2_sampled(np.arange(n))
    ex, ey, sx, sy = _sum64(x, y, m, 0.0)
    tol = (n + 16) * 2.0 ** -53
    ok = np.isfinite(ex) & np.isfinite(ey)
    assert ok.any()
    # the plain formula underflows to denormals at the far end; the mantissa path does not lose those bits
    tiny = 1e-290
    assert (np.abs(ax - ex)[ok] <= tol * sx[ok] + tiny).all()
    assert (np.abs(ay - ey)[ok] <= tol * sy[ok] + tiny).all()
    assert not np.isfinite(ax[~ok]).any() or not np.isfinite(ay[~ok]).any()


def test_sampled_sum_of_coincident_bodies(G):
    """eps = 0 and two bodies on one point: the term is inf * 0 as in the plain formula; with
    eps > 0 it is zero."""
    x, y, m = np.array([1.0, 1.0, 3.0]), np.array([2.0, 2.0, 2.5]), np.ones(3)
    ctx = G.GpuContext(G.GpuConfig(max_n=3))
    ctx.upload_bodies(G.Bodies.from_arrays(x, y, m))
    ctx.set_params(2, 0.0)
    ax, _ = ctx.n2_sampled([0, 1, 2])
    assert np.isnan(ax[0]) and np.isnan(ax[1]) and np.isfinite(ax[2])
    ctx.set_params(2, 0.5)
    ax, ay = ctx.n2_sampled([0, 1, 2])
    ex, ey, sx, sy = _sum64(x, y, m, 0.5)
    assert np.allclose(ax, ex, rtol=1e-15) and np.allclose(ay, ey, rtol=1e-15)


@pytest.mark.parametrize("n_idx", [1, 7, 300])
def test_sampled_sum_splits_its_bodies(G, n_idx):
    """Few samples over many bodies run several blocks a sample."""
    b = presets.plummer(20_011, seed=4)
    ctx = G.GpuContext(G.GpuConfig(max_n=len(b)))
    ctx.set_params(2, 0.01)
    ctx.upload_bodies(b)
    idx = np.linspace(0, len(b) - 1, n_idx).astype(np.int64)
    ax, ay = ctx.n2_sampled(idx)
    for k in range(0, n_idx, 37):
        dx, dy = b.x - b.x[idx[k]], b.y - b.y[idx[k]]
        f = b.mass * (dx * dx + dy * dy + 1e-4) ** -1.5
        s = np.abs(f * dx).sum() + np.abs(f * dy).sum()
        assert abs(ax[k] - (f * dx).sum()) <= 1e-14 * s and abs(ay[k] - (f * dy).sum()) <= 1e-14 * s


@pytest.mark.parametrize("n,n_max", [(1, 32), (17, 16), (33, 32), (500, 5), (1000, 16), (1001, 17), (3000, 32),
                                     (3000, 40), (2001, 64), (2500, 70)])
def test_fp64_near_field_rows_and_items(G, oracle, n, n_max):
    """REF forces against the oracle (1e-10 per body, the bound of the form)."""
    b = presets.uniform(n, seed=n)
    bounds = presets.BOUNDS["uniform"]
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, bounds, 4)
    ref = ob.copy()
    oracle.compute_fmm_force(ref, t, v, u, 4, eps, oracle.MODE_REF)
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4, eps64=eps))
    ctx.set_params(4, eps)
    ctx.build_tree(b, n_max, bounds)
    ax, ay = np.zeros(n), np.zeros(n)
    ctx.compute_forces(b.x, b.y, b.mass, ax, ay)
    assert (rel_vec_err(ax, ay, ref.ax, ref.ay) <= 1e-10).all()
