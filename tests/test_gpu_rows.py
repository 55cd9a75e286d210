"""Sorted rows (rows in warp items by length: a lane, four lanes or a warp to
a row) against the oracle, at the edges of the layout: lengths around the
class limits of small (16 / 64) and large (64 / 255) matrices, partial items,
empty rows, repeated columns, rectangular shapes, windows and the row counts
around them, and matrices that stay on the merge path.

Tolerances: FP64 rows within the oracle's row bound, FP32 rows within
(2*nnz_row + 3) * 2^-24 * sum|a_ij x_j|; power iterates within 1e-10 relative.
"""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pwm():
    import thesis_spmv_gb300 as t
    t.lib()
    return t


def _matrix(lengths, noc, seed):
    """Rows of the given lengths; columns anywhere, in any order, repeats too."""
    rng = np.random.default_rng(seed)
    lengths = np.asarray(lengths, np.int64)
    rs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    return O.CRSArrays(lengths.size, noc, rs, rng.integers(0, noc, int(rs[-1])).astype(np.int32),
                       rng.uniform(-1, 1, int(rs[-1])))


def _mixed(nor, seed, *kinds):
    """Rows drawn from the given lengths."""
    return np.random.default_rng(seed).choice(kinds, nor)


CASES = {
    "one_element": lambda: _matrix([1], 1, 1),
    "one_row": lambda: _matrix([900], 50, 2),
    "rows_31": lambda: _matrix([8] * 31, 70000, 3),
    "rows_32": lambda: _matrix([8] * 32, 70000, 4),
    "rows_33": lambda: _matrix([8] * 33, 70000, 5),
    "lane_limits": lambda: _matrix(_mixed(3001, 6, 11, 12, 13, 14, 15), 3001, 6),
    "small_limits": lambda: _matrix(_mixed(3001, 7, 14, 15, 16, 17, 62, 63, 64, 65), 3001, 7),
    "odd_even": lambda: _matrix(_mixed(4099, 8, 10, 11), 4099, 8),
    "empty_rows": lambda: _matrix(_mixed(5000, 9, 0, 0, 0, 12), 5000, 9),
    "longest_kept": lambda: _matrix([8] * 3000 + [1024], 3001, 10),
    "longest_past": lambda: _matrix([8] * 3000 + [1100], 3001, 11),  # the merge path
    "padding_past": lambda: _matrix([3] * 40000, 40000, 12),  # the merge path
    "wide": lambda: _matrix(_mixed(2000, 13, 5, 6, 30), 100000, 13),
    "tall": lambda: _matrix(_mixed(100000, 14, 4, 6), 700, 14),
    "large_limits": lambda: _matrix(_mixed(140000, 15, 62, 63, 64, 65), 140000, 15),
    "large_warp": lambda: _matrix(_mixed(45000, 16, 253, 254, 255, 256), 45000, 16),
    "rows_262143": lambda: _matrix(_mixed(262143, 17, 4, 8, 20), 262143, 17),
    "rows_262144": lambda: _matrix(_mixed(262144, 18, 4, 8, 20), 262144, 18),
    "windows_ragged": lambda: _matrix(np.where(np.arange(300001) < 40000, 40, _mixed(300001, 19, 0, 8, 10)), 300001, 19),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_spmv_rows(pwm, case):
    torch = pytest.importorskip("torch")
    A = CASES[case]()
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = np.random.default_rng(3).uniform(-1, 1, A.noc)
    want, bound = O.crs_mv(A, x), O.row_error_bound(A, x)
    y = np.full(A.nor, np.nan)
    M.mv(x, y)
    assert np.all(np.abs(y - want) <= bound)
    dx = torch.tensor(x, device="cuda")
    dy = torch.full((A.nor,), float("nan"), dtype=torch.float64, device="cuda")
    dx32, dy32 = dx.float(), dy.float()
    torch.cuda.synchronize()
    M.mv_device(dx.data_ptr(), dy.data_ptr())
    M.mv_device_f32(dx32.data_ptr(), dy32.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(dy.cpu().numpy(), y)
    s = O.crs_mv(O.CRSArrays(A.nor, A.noc, A.row_start, A.col_ind, np.abs(A.data)), np.abs(x))
    f32 = (2 * np.diff(A.row_start) + 3) * 2.0 ** -24 * s
    assert np.all(np.abs(dy32.cpu().numpy().astype(np.float64) - want) <= f32)
    rs, ci, d = M.getCSR()
    assert np.array_equal(rs, A.row_start) and np.array_equal(ci, A.col_ind) and np.array_equal(d, A.data)


def test_absent_elements_do_not_read_x(pwm):
    """Padding adds nothing, whatever x holds: infinities and NaNs reach
    exactly the rows that name them."""
    A = _matrix(_mixed(3000, 20, 9, 10, 15, 17, 70), 3000, 20)
    A.data = np.abs(A.data) + 0.5  # no inf - inf
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = np.random.default_rng(4).random(3000)
    x[[0, 1500, 2999]] = np.inf
    x[250] = np.nan
    y = np.zeros(3000)
    M.mv(x, y)
    want = O.crs_mv(A, x)
    assert np.array_equal(np.isnan(y), np.isnan(want)) and np.array_equal(np.isinf(y), np.isinf(want))


@pytest.mark.parametrize("it", [1, 2, 3, 4, 25])
@pytest.mark.parametrize("scale", [1.0, 1e150, 1e-150])
def test_power_steps(pwm, it, scale):
    A = _matrix(_mixed(5003, 21, 7, 8, 18, 70), 5003, 21)
    A.data = (np.abs(A.data) + 0.01) * scale
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x0 = np.random.default_rng(5).random(A.nor)
    xg, yg = x0.copy(), np.zeros(A.nor)
    M.powerIteration(xg, yg, it)
    xr, yr = O.power(A, x0, it)
    np.testing.assert_allclose(xg, xr, rtol=1e-10, atol=1e-13)
    np.testing.assert_allclose(yg, yr, rtol=1e-10, atol=1e-13)


def test_bits_do_not_depend_on_the_call(pwm):
    """The same bits from a plain and a captured launch, and in every run."""
    torch = pytest.importorskip("torch")
    A = _matrix(_mixed(270001, 22, 6, 9, 30), 270001, 22)
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = torch.rand(A.noc, dtype=torch.float64, device="cuda")
    y, z = torch.zeros(A.nor, dtype=torch.float64, device="cuda"), torch.zeros(A.nor, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    M.mv_device(x.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    M.set_stream(stream.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        M.mv_device(x.data_ptr(), z.data_ptr())
    for _ in range(3):
        z.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, z)
    M.set_stream(0)
