"""The exact sampled sum leaves the target out of its own sum, as a test of the index: a body
alone has no acceleration wherever it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 0.1])
@pytest.mark.parametrize("x", [3.0, np.inf, -np.inf, np.nan])
def test_a_body_alone(G, x, eps):
    ctx = G.GpuContext(G.GpuConfig(max_n=1, eps=0.0, eps64=eps))
    ctx.upload_bodies(G.Bodies.from_arrays([x], [1.0], [2.0]))
    ax, ay = ctx.n2_sampled([0])
    assert ax[0] == 0.0 and ay[0] == 0.0
