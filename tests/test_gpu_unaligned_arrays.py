"""Host arrays whose address is not a multiple of 8 (which numpy calls C-contiguous all the
same) give the bits that aligned ones give: they are copied, not read or written in place."""
import numpy as np
import pytest

from galax_gb300 import presets

pytestmark = pytest.mark.gpu
NAMES = ("x", "y", "vx", "vy", "mass", "ax", "ay")


def _array(G, n, pinned, keep):
    """n float64 at an address of 4 modulo 8, in ordinary or page-locked memory."""
    if pinned:
        keep.append(G.HostArray(n + 1))
        raw = keep[-1].array.view(np.uint8)
    else:
        raw = np.zeros(8 * n + 16, np.uint8)
        raw = raw[-raw.ctypes.data % 8:]
    a = raw[4:4 + 8 * n].view(np.float64)
    assert a.ctypes.data % 8 == 4 and a.flags.c_contiguous and not a.flags.aligned
    return a


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [1, 513, 70_001])
def test_unaligned_arrays(G, n, pinned):
    keep = []
    b = presets.uniform(n, seed=n)
    bounds = presets.BOUNDS["uniform"]
    u = G.Bodies(*[_array(G, n, pinned, keep) for _ in NAMES])
    for name in NAMES:
        getattr(u, name)[:] = getattr(b, name)
    ctx, ctu = (G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=3)) for _ in range(2))
    ctx.build_tree(b, 16, bounds)
    ctu.build_tree(u, 16, bounds)
    out = G.Bodies(*[_array(G, n, pinned, keep) for _ in NAMES])
    ctu.download_bodies(out)
    for name in NAMES:
        assert np.array_equal(getattr(u, name), getattr(b, name)) and np.array_equal(getattr(out, name), getattr(b, name))
    ax, ay = np.zeros(n), np.zeros(n)
    for _ in range(2):  # with the plan made, then with it there
        ctx.compute_forces(b.x, b.y, b.mass, ax, ay)
        ctu.compute_forces(u.x, u.y, u.mass, u.ax, u.ay)
        assert np.array_equal(u.ax, ax) and np.array_equal(u.ay, ay)
