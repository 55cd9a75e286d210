"""Triplet -> CRS by rows sorted in shared memory, at the sizes where its
paths change: rows of exactly 4096 entries (the longest it takes) and of 4097
(the radix sort), row groups that fill the 4096 keys exactly, row counts
around a CTA's 512, empty rows, repeated coordinates.  Bit-exact against a
stable sort on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lengths(kind, rng):
    if kind == "longest":
        n = np.zeros(700, np.int64)
        n[[0, 3, 4, 511, 512, 699]] = 4096
        return n
    if kind == "too_long":
        n = rng.integers(0, 9, 700)
        n[5] = 4097
        return n
    if kind == "groups_of_8":  # 512 rows fill the keys exactly
        return np.full(1024, 8)
    if kind == "groups_of_9":
        return np.full(1025, 9)
    if kind == "pairs":  # two rows fill the keys, three do not
        return np.full(13, 2048)
    if kind == "rows_511":
        return rng.integers(0, 20, 511)
    if kind == "rows_513":
        return rng.integers(0, 20, 513)
    return np.where(rng.random(5000) < 0.9, 0, rng.integers(1, 300, 5000))  # mostly empty


@pytest.mark.parametrize("repeat", [False, True])
@pytest.mark.parametrize("kind", ["longest", "too_long", "groups_of_8", "groups_of_9", "pairs", "rows_511", "rows_513",
                                  "mostly_empty"])
def test_rows(kind, repeat):
    torch = pytest.importorskip("torch")
    import thesis_spmv_gb300 as pwm
    rng = np.random.default_rng(3)
    n = _lengths(kind, rng)
    noc = 100 if repeat else 100_000
    r = np.repeat(np.arange(n.size), n).astype(np.int32)
    c = rng.integers(0, noc, r.size).astype(np.int32)
    v = rng.uniform(-1, 1, r.size)
    p = rng.permutation(r.size)
    r, c, v = r[p], c[p], v[p]
    q = np.lexsort((c, r))  # stable: equal coordinates keep their input order
    T = pwm.Triplet(n.size, noc, r.copy(), c.copy(), v.copy())
    H = pwm.CRSCuda(1)
    H.loadFromTriplets(T, 1)
    assert np.array_equal(T.row_coord, r[q]) and np.array_equal(T.col_coord, c[q])
    assert np.array_equal(T.data.view(np.uint64), v[q].view(np.uint64))
    dr, dc, dv = (torch.from_numpy(a).cuda() for a in (r, c, v))
    torch.cuda.synchronize()
    D = pwm.CRSCuda(1)
    D.loadFromDeviceTriplets(n.size, noc, r.size, dr.data_ptr(), dc.data_ptr(), dv.data_ptr())
    for M in (H, D):
        rs, ci, d = M.getCSR()
        assert np.array_equal(rs, np.concatenate([[0], np.cumsum(n)]))
        assert np.array_equal(ci, c[q]) and np.array_equal(d.view(np.uint64), v[q].view(np.uint64))
