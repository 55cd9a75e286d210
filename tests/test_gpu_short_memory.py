"""A load where device memory is short: what the handle cannot do without comes
first, and slices beside the merge plan only from what its other calls do not
need.  In a process of its own, with the rest of the memory held by torch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np, torch
import thesis_spmv_gb300 as pwm
from oracle import pyoracle as O
M = pwm.CRSCuda(1)
M.generatePoissonMatrix(8, 8, 1)
def leave(gb):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - int(gb * (1 << 30)), dtype=torch.uint8, device="cuda")
def fill():
    # what the library still finds, also in its own pool
    out = []
    try:
        while True:
            out.append(pwm.CRSCuda(1))
            out[-1].generatePoissonMatrix(1024, 1024, 1)
    except RuntimeError:
        return out
def check(m):
    n = m * m
    x = np.random.default_rng(1).random(n).reshape(m, m)
    y = np.full(n, np.nan)
    M.mv(x.reshape(-1), y)
    p = np.zeros((m + 2, m + 2))
    p[1:-1, 1:-1] = x
    want = 4 * x - p[:-2, 1:-1] - p[2:, 1:-1] - p[1:-1, :-2] - p[1:-1, 2:]
    assert np.all(np.abs(y.reshape(m, m) - want) <= 16 * 2.0 ** -53 * 8)
"""


def _run(body):
    r = subprocess.run([sys.executable, "-c", HEAD + body + "\nprint('ok')"], capture_output=True, text=True, timeout=600,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-4000:]


def test_a_load_that_fits_without_slices():
    """4096^2 stencil: 1.0 GiB of CRS arrays and 1.0 of merge plan while it is
    built, 0.7 of slices.  With 2.4 GiB left the slices do not fit beside them:
    the load goes on without, and products and power steps have their memory."""
    _run("""
hog = leave(2.4)
M.generatePoissonMatrix(4096, 4096, 1)
assert M.layout() == "merge"
check(4096)
x, y = np.random.default_rng(2).random(4096 * 4096), np.zeros(4096 * 4096)
M.powerIteration(x, y, 3)
assert np.all(np.isfinite(y)) and abs(np.linalg.norm(y) - 1) < 1e-12
del hog
torch.cuda.empty_cache()
M.generatePoissonMatrix(4096, 4096, 1)
assert M.layout() == "diagonals"
check(4096)
""")


def test_buffers_that_grow_where_memory_is_short():
    """One handle, ever larger matrices: a buffer asks for twice the room of
    the one it replaces, and is content with what it needs.  8192^2 rows after
    6500^2: vectors of 0.5 GiB each, where twice the room were 0.63."""
    _run("""
M.generatePoissonMatrix(6500, 6500, 1)
check(6500)
M.generatePoissonMatrix(8, 8, 1)
check(8)
# 8192^2: 4.0 GiB of CRS arrays, 4.3 of plan while it is built
hog = leave(8.9)
M.generatePoissonMatrix(8192, 8192, 1)
check(8192)
""")


def test_a_failed_load_leaves_the_memory_and_the_handle():
    """Too little memory for the plan: an error, not a crash, and all that the
    load had taken is back: the next, smaller one fits."""
    _run("""
hog = leave(1.5)
for _ in range(3):
    try:
        M.generatePoissonMatrix(4096, 4096, 1)
        raise SystemExit("the load should not have fitted")
    except RuntimeError:
        pass
    M.generatePoissonMatrix(2048, 2048, 1)
    check(2048)
""")


@pytest.mark.parametrize("then", ["the same product", "a small product"])
def test_vectors_that_do_not_fit(then):
    """The load fits, the vectors of a host-array product (0.37 GiB each: ten rows
    of 50 M columns) do not: an error, and the handle's next products have
    vectors again."""
    _run("""
check(8)
def wide():
    M.loadCSR(10, 50_000_000, np.arange(11, dtype=np.int32), np.arange(10, dtype=np.int32) * 4_999_999, np.ones(10))
def product():
    x, y = np.arange(50_000_000) % 1000 * 1.0, np.full(10, np.nan)
    M.mv(x, y)
    assert np.array_equal(y, x[np.arange(10) * 4_999_999])
wide()
hog = leave(0.15)
others = fill()
try:
    product()
    raise SystemExit("the vectors should not have fitted")
except RuntimeError:
    pass
""" + ("""
del others, hog
torch.cuda.empty_cache()
product()
""" if then == "the same product" else """
M.generatePoissonMatrix(8, 8, 1)
check(8)
"""))
