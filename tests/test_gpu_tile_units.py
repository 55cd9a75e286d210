"""The blocked formats' tile kernel on diagonal tiles: tiles of 1 to 4
diagonals share one staged x window (one unit per diagonal), tiles of 5 keep
their rows together, border tiles hold diagonals of a few elements, windows
and rows end raggedly, and x starts off a 16-byte boundary (no bulk copy).

Tolerance: each row within the oracle's row bound.
"""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

CASES = [
    (300, [0]), (300, [-1, 0, 1]), (1024, [-2, -1, 0, 1]), (1025, [-2, -1, 0, 1, 2]), (20011, [-141, -1, 0, 1, 141]),
    (70001, [-1024, -1, 0, 1, 1024]), (70001, [-513, -512, -511, 0, 511, 512, 513]), (160003, [-64, 0, 64]),
    (1300001, [-1500, -1, 0, 1, 1500]),
]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("fmt", ["csb", "coh"])
@pytest.mark.parametrize("n,offsets", CASES)
def test_diagonal_tiles(n, offsets, fmt, shift):
    torch = pytest.importorskip("torch")
    import thesis_spmv_gb300 as pwm
    rng = np.random.default_rng(n + len(offsets))
    cols = np.arange(n)[:, None] + np.array(offsets)[None, :]
    keep = (cols >= 0) & (cols < n)
    rs = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    ci = cols[keep].astype(np.int32)
    A = O.CRSArrays(n, n, rs, ci, rng.uniform(-1, 1, ci.size))
    M = pwm.CSBCuda() if fmt == "csb" else pwm.COHCuda()
    M.loadCSR(n, n, rs, ci, A.data)
    x = rng.uniform(-1, 1, n)
    dx = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
    dx[shift:shift + n] = torch.from_numpy(x).cuda()
    dy = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for v in (range(4) if fmt == "csb" else [None]):
        if v is not None:
            M.set_csb_variant(v)
        M.mv_device(dx.data_ptr() + 8 * shift, dy.data_ptr())
        torch.cuda.synchronize()
        assert np.all(np.abs(dy.cpu().numpy() - O.crs_mv(A, x)) <= O.row_error_bound(A, x))
