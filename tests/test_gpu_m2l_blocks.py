"""M2L and its transpose at p = 8 in FP32, four units a block: unit counts that fill the last
block by one to four, against the FP64 form of the same lists."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [7, 8, 9])
@pytest.mark.parametrize("n,n_max", [(9, 1), (40, 4), (41, 4), (45, 4), (50, 4), (333, 8), (5_003, 16)])
def test_mixed_against_fp64(G, n, n_max, p):
    """Within 1e-4 of the rms value (rounding 6e-8 through the 2p + 1 orders of the recurrence,
    times the sizes of the terms over their sum)."""
    b = presets.uniform(n, seed=n)
    lam = np.random.default_rng(n).standard_normal((2, n))
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=p, eps64=0.5))
    ctx.build_tree(b, n_max, presets.BOUNDS["uniform"])
    ctx.upload_bodies(b)
    got = []
    for prec in (G.PREC_FP64, G.PREC_MIXED):
        ctx.set_mode(G.MODE_ACCURATE, prec, 0.5)
        o = G.Bodies.new(n)
        ctx.forces_resident()
        ctx.download_bodies(o)
        got.append([o.ax, o.ay, *(ctx.force_vjp(*lam) if p <= 8 else ())])  # the adjoint goes to p = 8
    assert ctx.plan_info()[0] > 0
    for a, m in zip(*got):
        assert np.abs(m - a).max() <= 1e-4 * np.sqrt(np.mean(a ** 2))
