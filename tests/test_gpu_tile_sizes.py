"""The tile kernel of the blocked formats at sizes between one round of resident
CTAs and the next: windows of 64 to 1024 rows, 7 or 8 CTAs per SM, units
shorter than a CTA.  Every variant against the oracle's row bound, and the time
of mid-size stencils, whose units once left most warps idle."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def _irregular(n, seed):
    rng = np.random.default_rng(seed)
    lens = np.clip(rng.lognormal(1.5, 1.0, n).astype(np.int64), 1, 400)
    rs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    k = int(rs[-1])
    near = rng.random(k) < 0.6
    ci = np.where(near, np.clip(np.repeat(np.arange(n), lens) + rng.integers(-900, 901, k), 0, n - 1), rng.integers(0, n, k))
    return O.CRSArrays(n, n, rs, ci.astype(np.int32), rng.uniform(-1, 1, k))


# rows: windows of 64 in 1 round of 7 CTAs (7 * 152 windows), in 1 of 8, past
# both; of 128, 256, 512 at 8 and at 7; of 1024 at 8 and at 7
ROWS = [1064 * 64, 1065 * 64, 1216 * 64 - 3, 1217 * 64, 2200 * 64, 1100 * 256, 1300 * 256, 2300 * 512 + 7, 1300 * 1024]


@pytest.mark.parametrize("kind", ["stencil", "irregular"])
@pytest.mark.parametrize("fmt", ["csb", "coh"])
@pytest.mark.parametrize("rows", ROWS)
def test_rows(rows, fmt, kind):
    import thesis_spmv_gb300 as pwm
    if kind == "irregular" and rows > 400_000:
        pytest.skip("covered by the smaller ones: the flat units do not depend on the window")
    m = int(rows ** 0.5)
    A = O.fill_poisson(m, rows // m) if kind == "stencil" else _irregular(rows, 3)
    A.data = np.random.default_rng(1).uniform(-1, 1, A.data.size)
    M = (pwm.CSBCuda if fmt == "csb" else pwm.COHCuda)(4)
    M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
    x = np.random.default_rng(2).uniform(-1, 1, A.noc)
    want, bound = O.crs_mv(A, x), O.row_error_bound(A, x)
    for v in range(4):
        M.set_csb_variant(v)
        y = np.full(A.nor, np.nan)
        M.mv(x, y)
        assert np.all(np.abs(y - want) <= bound)


def _us(rows):
    torch = pytest.importorskip("torch")
    import thesis_spmv_gb300 as pwm
    m = int(rows ** 0.5)
    M = pwm.CSBCuda(1)
    M.generatePoissonMatrix(m, rows // m, 1)
    M.set_stream(torch.cuda.current_stream().cuda_stream)
    n = M.dims()[0]
    x, y = torch.rand(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    best = 1e9
    for _ in range(6):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        for _ in range(40):
            M.mv_device(x.data_ptr(), y.data_ptr())
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) * 25)
    return best


@pytest.mark.parametrize("rows,share", [(290_000, 0.75), (560_000, 0.9), (1_150_000, 1.1)])
def test_mid_size_stencils_take_their_share(rows, share):
    """Beside 1.5 M rows (29 us): 290 000 rows 16 us, 560 000 20 us and 1.15 M
    23 us; with idle warps and a round more 27, 31 and 39."""
    assert _us(rows) <= share * _us(1_500_000)
