"""Diagonal slices (rows in slices of 64, one column - row offset per slot)
against the oracle, at the edges of the layout: groups of 5 slots and their
remainders, partial last slices, masked slots at the matrix border, repeated
and descending columns, empty rows, rectangular shapes, one and several
slices per warp.

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


def _diagonals(nor, noc, offsets, seed, drop=0.0, descending=False):
    """Rows with columns i + o for o in offsets (kept with probability
    1 - drop, where inside the matrix), in the order of the offsets."""
    rng = np.random.default_rng(seed)
    offs = np.array(sorted(offsets, reverse=descending), np.int64)
    cols = np.arange(nor)[:, None] + offs[None, :]
    keep = (cols >= 0) & (cols < noc) & (rng.random(cols.shape) >= drop)
    rs = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    ci = cols[keep].astype(np.int32)
    return O.CRSArrays(nor, noc, rs, ci, rng.uniform(-1, 1, ci.size))


CASES = {
    "one_row": lambda: _diagonals(1, 1, [0], 1),
    "rows_63": lambda: _diagonals(63, 63, [-1, 0, 1], 2),
    "rows_64": lambda: _diagonals(64, 64, [-1, 0, 1], 3),
    "rows_65": lambda: _diagonals(65, 65, [-1, 0, 1], 4),
    "slots_4": lambda: _diagonals(5000, 5000, [-7, -1, 0, 900], 5),
    "slots_5": lambda: _diagonals(5000, 5000, [-900, -1, 0, 1, 900], 6),
    "slots_6": lambda: _diagonals(5000, 5000, range(6), 7),
    "slots_10": lambda: _diagonals(5000, 5000, range(-4, 6), 8),
    "slots_11": lambda: _diagonals(5000, 5000, range(-5, 6), 9),
    "slots_33": lambda: _diagonals(7001, 7001, range(-16, 17), 10),
    "slots_256": lambda: _diagonals(4000, 4000, range(-128, 128), 11),
    "slots_257": lambda: _diagonals(4000, 4000, range(-128, 129), 12),  # past the limit: the merge layout
    "partial_rows": lambda: _diagonals(20011, 20011, [-141, -1, 0, 1, 141], 13, drop=0.1),
    "too_sparse": lambda: _diagonals(20011, 20011, range(9), 14, drop=0.5),  # padding past a quarter: merge
    "repeated": lambda: _diagonals(3000, 3000, [-2, 0, 0, 3], 15),
    "descending": lambda: _diagonals(3000, 3000, [-40, -1, 0, 1, 40], 16, descending=True),
    "wide": lambda: _diagonals(3000, 9000, [0, 1, 3000, 8999], 17),
    "tall": lambda: _diagonals(9000, 3000, [-5999, -1, 0, 1], 18),  # rows past the band are empty
    "several_per_warp": lambda: _diagonals(700001, 700001, [-1201, -1, 0, 1, 1201], 19),
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


@pytest.mark.parametrize("drop", [0.0, 0.1])
def test_absent_elements_do_not_read_x(pwm, drop):
    """A slot's missing elements add nothing, whatever x holds at their
    column: infinities and NaNs reach exactly the rows that name them."""
    A = _diagonals(1000, 1000, [-31, -1, 0, 1, 31], 21, drop=drop)
    A.data = np.abs(A.data) + 0.5  # no inf - inf
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = np.random.default_rng(4).random(1000)
    x[[0, 500, 999]] = np.inf
    x[250] = np.nan
    y = np.zeros(1000)
    M.mv(x, y)
    want = O.crs_mv(A, x)
    assert np.array_equal(np.isnan(y), np.isnan(want)) and np.array_equal(np.isinf(y), np.isinf(want))


@pytest.mark.parametrize("it", [1, 2, 3, 4, 25])
@pytest.mark.parametrize("scale", [1.0, 1e150, 1e-150])
def test_power_steps(pwm, it, scale):
    A = _diagonals(5003, 5003, [-70, -1, 0, 1, 70], 22)
    A.data = (np.abs(A.data) + 0.01) * scale
    M = pwm.CRSCuda(1)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x0 = np.random.default_rng(5).random(A.nor)
    xg, yg = x0.copy(), np.zeros(A.nor)
    M.powerIteration(xg, yg, it)
    xr, yr = O.power(A, x0, it)
    np.testing.assert_allclose(xg, xr, rtol=1e-10, atol=1e-13)
    np.testing.assert_allclose(yg, yr, rtol=1e-10, atol=1e-13)


def test_a_handle_reloaded_with_another_kind(pwm):
    """Stencil, irregular, stencil in one handle: each load's own layout."""
    M = pwm.CRSCuda(1)
    rng = np.random.default_rng(6)
    n = 6000
    cols = np.sort(rng.integers(0, n, (n, 5)), axis=1).astype(np.int32)
    B = O.CRSArrays(n, n, (5 * np.arange(n + 1)).astype(np.int32), cols.reshape(-1), rng.uniform(-1, 1, 5 * n))
    for A in (CASES["slots_5"](), B, CASES["slots_11"]()):
        M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
        x = rng.uniform(-1, 1, A.noc)
        y = np.zeros(A.nor)
        M.mv(x, y)
        assert np.all(np.abs(y - O.crs_mv(A, x)) <= O.row_error_bound(A, x))


@pytest.mark.parametrize("steps,graph", [(2, True), (3, True), (4, False), (8, True)])
def test_service_batches(pwm, steps, graph):
    """The serving loop's diagonal-slice classes: matrices of 1 .. 300 slices,
    3 .. 11 slots, in every precision, beside one that does not fit the
    layout.  Rounds of 2 and 3 steps have no or one key step.  Each solve's
    eigenpair against the oracle, and the same bits alone as in the mix."""
    from thesis_spmv_gb300.service import Service
    mats = []
    for k, (n, offs) in enumerate([(40, [-1, 0, 1]), (64, [-8, -1, 0, 1, 8]), (1000, range(-5, 6)),
                                   (19000, [-137, -1, 0, 1, 137])]):
        A = _diagonals(n, n, offs, 40 + k)
        A.data = np.abs(A.data) + 0.05
        mid = A.row_start[n // 2] + int(np.argmin(np.abs(A.col_ind[A.row_start[n // 2]:A.row_start[n // 2 + 1]] - n // 2)))
        A.data[mid] += 12.0  # a dominant, well separated eigenvalue
        mats.append(A)
    rng = np.random.default_rng(7)
    n = 800
    cols = np.sort(np.argsort(rng.random((n, n)), axis=1)[:, :6], axis=1).astype(np.int32)
    mats.append(O.CRSArrays(n, n, (6 * np.arange(n + 1)).astype(np.int32), cols.reshape(-1), rng.uniform(0.1, 1, 6 * n)))

    def run(which):
        svc = Service(hbm_budget_bytes=1 << 30, round_iterations=steps, use_graph=graph)
        ids = []
        for i, prec in which:
            x0 = np.random.default_rng(100 + i).random(mats[i].nor)
            tol = 1e-5 if prec == pwm.PREC_F32 else 1e-10
            ids.append(svc.submit_csr(mats[i], max_it=6000, tol=tol, precision=prec, x0=x0, keep_vector=True))
        svc.run_until_idle()
        return [svc.result(i, want_vector=True) for i in ids]

    which = [(i, p) for i in range(len(mats)) for p in (pwm.PREC_F64, pwm.PREC_F32, pwm.PREC_MIXED)]
    for (i, prec), (r, u) in zip(which, run(which)):
        assert r.converged == 1
        lam, res = O.rayleigh(mats[i], u)
        assert res <= (1e-4 if prec == pwm.PREC_F32 else 2e-10)
        assert abs(r.lambda_ - lam) <= (1e-5 if prec == pwm.PREC_F32 else 1e-10) * abs(lam)
        if i in (0, 3):
            (ra, ua), = run([(i, prec)])
            assert ra.iterations == r.iterations and ra.lambda_ == r.lambda_
            assert np.array_equal(ua.view(np.uint64), u.view(np.uint64))
