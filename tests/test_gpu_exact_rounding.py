"""The rounding of the mixed form over the reference's lists.  Their pairs may be closer than the
nodes are wide, so the series' terms grow with the order and what M2L's recurrence rounds away
decides the error."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu
# geometric mean of the errors below with every derivative order's coefficients formed from dx, dy
# and 1/R^2 (3 presets, 5 orders, 24 seeds: 5 % standard error); formed from dx / R^2 and dy / R^2,
# whose rounding is common to all orders, it is 3.1e-6
PER_ORDER = 2.57e-6


def test_exact_mixed_against_fp64(G):
    n, logs = 4001, []
    for preset in ("plummer", "uniform", "disk"):
        for seed in range(100, 124):
            b = presets.make(preset, n, seed=seed)
            ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=4))
            ctx.build_tree(b, 16, presets.BOUNDS[preset])
            ctx.upload_bodies(b)
            eps = max(presets.cli_softening(b.x, b.y), 1e-3)
            for p in range(4, 9):
                ctx.set_params(p, eps)
                a = []
                for prec in (G.PREC_FP64, G.PREC_MIXED):
                    ctx.set_mode(G.MODE_EXACT, prec, 0.5)
                    ctx.forces_resident()
                    o = G.Bodies.new(n)
                    ctx.download_bodies(o)
                    a.append(np.stack([o.ax, o.ay]))
                logs.append(0.5 * np.log((2 * (a[1] - a[0]) ** 2).mean() / (a[0] ** 2).mean()))
            ctx.close()
    assert np.exp(np.mean(logs)) <= 1.1 * PER_ORDER
