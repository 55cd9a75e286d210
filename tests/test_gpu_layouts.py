"""Which layout a matrix's products run on, at the rules' edges, with the
values against the oracle: diagonal slices, sorted rows, the merge path and
SELL-32, each reached and each refused.  A launch variant asked for puts the
handle on the merge kernels; the slices' products against those on the same
matrix, and no slower than they.

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


def _rows(lengths, noc, seed, band=0):
    """Rows of the given lengths; columns anywhere or within `band` of the diagonal."""
    rng = np.random.default_rng(seed)
    rs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    k = int(rs[-1])
    if band:
        ci = np.repeat(np.arange(len(lengths)), lengths) + rng.integers(-band, band + 1, k)
        ci = np.clip(ci, 0, noc - 1)
    else:
        ci = rng.integers(0, noc, k)
    return O.CRSArrays(len(lengths), noc, rs, ci.astype(np.int32), rng.uniform(-1, 1, k))


def _diagonals(n, offsets, seed, drop=0.0):
    rng = np.random.default_rng(seed)
    cols = np.arange(n)[:, None] + np.array(sorted(offsets))[None, :]
    keep = (cols >= 0) & (cols < n) & (rng.random(cols.shape) >= drop)
    rs = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return O.CRSArrays(n, n, rs, cols[keep].astype(np.int32), rng.uniform(-1, 1, int(rs[-1])))


# kind: matrix, layout in FP64, layout in FP32
CASES = {
    "stencil": (lambda: O.fill_poisson(200, 100), "diagonals", "diagonals"),
    "slots_256": (lambda: _diagonals(4000, range(-128, 128), 1), "diagonals", "diagonals"),
    "slots_257": (lambda: _diagonals(4000, range(-128, 129), 2), "rows", "rows"),
    # 64 stored elements per slot against 1.25 nnz + 128 slots
    "diagonal_padding_kept": (lambda: _diagonals(20_000, range(9), 3, drop=0.15), "diagonals", "diagonals"),
    "diagonal_padding_past": (lambda: _diagonals(20_000, range(9), 4, drop=0.5), "rows", "rows"),
    "irregular": (lambda: _rows(np.random.default_rng(5).integers(5, 40, 20_000), 20_000, 5), "rows", "rows"),
    # the longest row against 1024 + nnz / 1000
    "longest_kept": (lambda: _rows([8] * 3000 + [1024], 3001, 6), "rows", "rows"),
    "longest_past": (lambda: _rows([8] * 3000 + [1100], 3001, 7), "merge", "merge"),
    # rows of 3 store 4: 4 n against 3.75 n + 16384
    "row_padding_kept": (lambda: _rows([3] * 60_000, 60_000, 8), "rows", "rows"),
    "row_padding_past": (lambda: _rows([3] * 80_000, 80_000, 9), "merge", "merge"),
    # 2 n / 64 items of one unit each, past 65 536 of them
    "short_items": (lambda: _rows([2] * 2_200_000, 2_200_000, 10), "merge", "merge"),
    # narrow columns: past 8192 items of fewer than 6 units; every row as long
    # as the next, so FP32 runs on SELL-32
    "short_narrow_items": (lambda: _rows([6] * 280_000, 280_000, 11, band=150), "merge", "sell"),
    "few_narrow_items": (lambda: _rows([6] * 250_000, 250_000, 12, band=150), "rows", "rows"),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_layout(pwm, case):
    torch = pytest.importorskip("torch")
    make, fp64, fp32 = CASES[case]
    A = make()
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    assert M.layout() == fp64
    x = np.random.default_rng(3).uniform(-1, 1, A.noc)
    want, bound = O.crs_mv(A, x), O.row_error_bound(A, x)
    y = np.full(A.nor, np.nan)
    M.mv(x, y)
    assert np.all(np.abs(y - want) <= bound)
    x32 = torch.tensor(x, dtype=torch.float32, device="cuda")
    y32 = torch.full((A.nor,), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    M.mv_device_f32(x32.data_ptr(), y32.data_ptr())
    torch.cuda.synchronize()
    assert M.layout(pwm.PREC_F32) == fp32
    s = O.crs_mv(O.CRSArrays(A.nor, A.noc, A.row_start, A.col_ind, np.abs(A.data)), np.abs(x))
    f32 = (2 * np.diff(A.row_start) + 3) * 2.0 ** -24 * s
    assert np.all(np.abs(y32.cpu().numpy().astype(np.float64) - want) <= f32)
    # the merge kernels on the same matrix
    M.set_launch_variant(0)
    assert M.layout() == "merge"
    z = np.full(A.nor, np.nan)
    M.mv(x, z)
    assert np.all(np.abs(z - want) <= bound)
    if fp64 == "merge":
        assert np.array_equal(y, z)
    # a load chooses anew
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    assert M.layout() == fp64
    M.mv(x, z)
    assert np.array_equal(y, z)


@pytest.mark.parametrize("kind", ["stencil", "irregular"])
def test_power_and_chunked_products_on_both_layouts(pwm, kind):
    """600 x 700 grid and 300 001 irregular rows: host-array products in 16
    chunks, power steps, before and after the handle moves to the merge
    kernels, bits equal to the device-resident product on either."""
    torch = pytest.importorskip("torch")
    A = O.fill_poisson(600, 700) if kind == "stencil" else _rows(
        np.random.default_rng(6).integers(5, 30, 300_001), 300_001, 13)
    A.data = np.abs(A.data) + 0.01  # a dominant Perron eigenvalue
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = np.random.default_rng(7).random(A.noc)
    dx, dy = torch.tensor(x, device="cuda"), torch.empty(A.nor, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    xr, yr = O.power(A, x, 7)
    for layout in ("diagonals" if kind == "stencil" else "rows", "merge"):
        if layout == "merge":
            M.set_launch_variant(1)
        assert M.layout() == layout
        y = np.full(A.nor, np.nan)
        M.mv(x, y)
        assert np.all(np.abs(y - O.crs_mv(A, x)) <= O.row_error_bound(A, x))
        M.mv_device(dx.data_ptr(), dy.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(dy.cpu().numpy(), y)
        xg, yg = x.copy(), np.zeros(A.nor)
        M.powerIteration(xg, yg, 7)
        np.testing.assert_allclose(xg, xr, rtol=1e-10, atol=1e-13)
        np.testing.assert_allclose(yg, yr, rtol=1e-10, atol=1e-13)


def _us(M, x, y):
    import torch
    best = 1e9
    for _ in range(6):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        for _ in range(20):
            M.mv_device(x.data_ptr(), y.data_ptr())
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) * 50)
    return best


@pytest.mark.parametrize("lengths", ["9000_last", "17000_last", "8_of_10000", "stencil"])
def test_no_slower_than_the_merge_kernels(pwm, lengths):
    """The layout a load chooses against the merge kernels in the variant the
    tuner chose for the same handle (10 % for noise)."""
    torch = pytest.importorskip("torch")
    n = 1 << 20
    M = pwm.CRSCuda(1)
    if lengths == "stencil":
        M.generatePoissonMatrix(1024, 1024, 1)
    else:
        rows = {"9000_last": [16] * (n - 1) + [9000], "17000_last": [16] * (n - 1) + [17_000],
                "8_of_10000": [9] * (n - 8) + [10_000] * 8}[lengths]
        A = _rows(rows, n, 14)
        M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    M.set_stream(torch.cuda.current_stream().cuda_stream)
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y = torch.empty(n, dtype=torch.float64, device="cuda")
    chosen = _us(M, x, y)
    M.set_launch_variant(M.launch_variant() & ~2)
    assert M.layout() == "merge"
    assert chosen <= 1.1 * _us(M, x, y)
