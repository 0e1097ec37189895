"""Plans around the sizes where their scans change from one block to a cluster (4,096
entries), and P2L as a stream over ragged leaves, against the oracle."""
import numpy as np
import pytest

from galax_gb300 import presets
from helpers import oracle_case, rel_vec_err
from test_gpu_near_split import _gpu, _oracle_wx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_max", [(4095 * 3, 3), (4096 * 3, 3), (4096 * 3 + 1, 3), (13_001, 1)])
def test_plan_at_the_scan_sizes(G, oracle, n, n_max):
    """4,095, 4,096, 4,097 and 13,001 leaves: forces within 1e-10 of the oracle's evaluation of
    its own lists (one pair more or less is 1e-4 and above), and its pair counts."""
    p, theta, theta_w = 3, 0.5, 0.4
    b = presets.uniform(n, seed=n)
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, presets.BOUNDS["uniform"], p)
    assert t.n_leaves == -(-n // n_max)
    ref, far, p2p, m2p, p2l = _oracle_wx(oracle, ob, t, theta, theta_w, p, eps)
    ax, ay, info = _gpu(G, ob, t, v, u, p, eps, G.PREC_FP64, theta, theta_w)
    assert rel_vec_err(ax, ay, ref.ax, ref.ay).max() < 1e-10
    assert info[0][0] == far.off[-1] and info[1] == (m2p.off[-1], p2l.off[-1])


@pytest.mark.parametrize("n,n_max,p", [(10_007, 13, 6), (10_007, 13, 8), (9_001, 32, 7), (33, 32, 6)])
def test_p2l_stream_on_ragged_leaves(G, oracle, n, n_max, p):
    """FP64 within 1e-10 per body; mixed within 1e-4 of the rms acceleration (rounding 6e-8
    through the 2p + 1 orders of the recurrence, times the sizes of the terms over their sum)."""
    theta, theta_w = 0.5, 0.4
    b = presets.plummer(n, seed=n)
    ob, t, v, u, eps = oracle_case(oracle, b, n_max, presets.BOUNDS["plummer"], p)
    ref, *_ = _oracle_wx(oracle, ob, t, theta, theta_w, p, eps)
    ax, ay, _ = _gpu(G, ob, t, v, u, p, eps, G.PREC_FP64, theta, theta_w)
    assert rel_vec_err(ax, ay, ref.ax, ref.ay).max() < 1e-10
    ax, ay, _ = _gpu(G, ob, t, v, u, p, eps, G.PREC_MIXED, theta, theta_w)
    rms = np.sqrt(np.mean(ref.ax ** 2 + ref.ay ** 2))
    assert np.hypot(ax - ref.ax, ay - ref.ay).max() <= 1e-4 * rms
