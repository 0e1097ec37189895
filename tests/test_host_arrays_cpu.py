"""Which host arrays the kernels may read and write in place, and that a call has read its
arrays when it returns: the library's host side over a stand-in for the CUDA runtime
(fake_cudart.c), without a GPU."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {root!r})
import galax_gb300 as G
fake = C.CDLL({fake!r})
count = lambda name: C.c_long.in_dll(fake, name).value
fail = C.c_size_t.in_dll(fake, "fake_fail_bytes")

def array(n, shift):
    "n float64 zeros, shift bytes past an address that is a multiple of 8"
    a = np.frombuffer(bytearray(8 * n + 16), np.uint8)
    a = a[-a.ctypes.data % 8 + shift:][:8 * n].view(np.float64)
    assert a.ctypes.data % 8 == shift and a.flags.c_contiguous
    return a

def bodies(n, shift=0):
    return G.Bodies(*[array(n, shift) for _ in range(7)])
"""


@pytest.fixture(scope="module")
def run(G, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)

    def go(body):
        code = PRELUDE.format(root=os.path.dirname(HERE), fake=so) + body
        r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "LD_PRELOAD": so}, capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr
    return go


@pytest.mark.parametrize("shift", [1, 4, 7])
def test_unaligned_arrays_are_copied(run, shift):
    """A double's address must be a multiple of 8 for a kernel to load or store it there: other
    arrays take the copies, any of the seven and in both directions."""
    run(f"""
n = 1000
ctx = G.GpuContext(G.GpuConfig(max_n=n))
c = count("fake_copies")
ctx.upload_bodies(bodies(n))
ctx.download_bodies(bodies(n))
assert count("fake_copies") == c                      # in place
ctx.upload_bodies(bodies(n, {shift}))
assert count("fake_copies") == c + 7
ctx.download_bodies(bodies(n, {shift}))
assert count("fake_copies") == c + 14
for k in range(7):
    b = bodies(n)
    setattr(b, ("x", "y", "vx", "vy", "mass", "ax", "ay")[k], array(n, {shift}))
    c = count("fake_copies")
    ctx.upload_bodies(b)
    ctx.download_bodies(b)
    assert count("fake_copies") == c + 14, k
ids = np.frombuffer(bytearray(8 * n + 16), np.uint8)
ids = ids[-ids.ctypes.data % 8 + {shift}:][:8 * n].view(np.int64)
c = count("fake_copies")
ctx._check(G.lib().gx_body_ids(ctx._h, G._p(ids, G._I64)))
assert count("fake_copies") == c + 1
""")


def test_a_failed_upload_has_read_its_arrays(run):
    """An upload that fails behind its kernel (no memory for the ids) waits before it returns:
    the caller may free the arrays then."""
    run("""
n = 1000
ctx = G.GpuContext(G.GpuConfig(max_n=n))
fail.value = 4 * n + 4 * n // 8                       # the ids, with gx_ensure's eighth
w, c = count("fake_waits"), count("fake_copies")
try:
    ctx.upload_bodies(bodies(n))
    raise SystemExit("the upload did not fail")
except G.GpuError as e:
    assert e.code == 3, e
assert count("fake_copies") == c and count("fake_waits") == w + 1
fail.value = 0
ctx.upload_bodies(bodies(n))
assert count("fake_waits") == w + 2
""")


def test_large_uploads_do_not_look_at_the_pages(run):
    """Above the kernel copy's limit the arrays are copied whatever they are: their pages are
    neither asked after nor touched."""
    run("""
n = 262_145
ctx = G.GpuContext(G.GpuConfig(max_n=n))
b = bodies(n)
q, c = count("fake_queries"), count("fake_copies")
ctx.upload_bodies(b)
ctx.download_bodies(b)
assert count("fake_queries") == q and count("fake_copies") == c + 14
""")
