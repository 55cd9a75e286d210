"""The first FP32 product of a handle: its FP32 values are made in that call,
and the kernel that reads them starts its loads before the kernel before it on
the stream has ended.  Fresh handles, the conversion and the product right
behind each other (and behind other work on the stream): the first product has
the bits of the later ones, and its rows lie within (2*nnz_row + 3) * 2^-24 *
sum|a_ij x_j| of the FP64 oracle."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def _irregular(n):
    rng = np.random.default_rng(n)
    rs = np.concatenate([[0], np.cumsum(rng.integers(8, 40, n))]).astype(np.int32)
    return O.CRSArrays(n, n, rs, rng.integers(0, n, int(rs[-1])).astype(np.int32), rng.uniform(-1, 1, int(rs[-1])))


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("kind", ["one_slice", "stencil", "large_stencil", "irregular"])
def test_first_fp32_product(kind, busy):
    torch = pytest.importorskip("torch")
    import thesis_spmv_gb300 as pwm
    A = {"one_slice": lambda: O.fill_poisson(8, 8), "stencil": lambda: O.fill_poisson(300, 211),
         "large_stencil": lambda: O.fill_poisson(1201, 1103), "irregular": lambda: _irregular(30011)}[kind]()
    A.data = np.random.default_rng(1).uniform(-1, 1, A.data.size)
    x = np.random.default_rng(2).uniform(-1, 1, A.noc)
    want = O.crs_mv(A, x)
    s = O.crs_mv(O.CRSArrays(A.nor, A.noc, A.row_start, A.col_ind, np.abs(A.data)), np.abs(x))
    bound = (2 * np.diff(A.row_start) + 3) * 2.0 ** -24 * s
    dx = torch.tensor(x, dtype=torch.float32, device="cuda")
    first = torch.empty(A.nor, dtype=torch.float32, device="cuda")
    later = torch.empty_like(first)
    z = torch.ones(1 << 24, device="cuda")
    torch.cuda.synchronize()
    for _ in range(8):
        M = pwm.CRSCuda(1)
        M.loadCSR(A.nor, A.noc, A.row_start, A.col_ind, A.data)
        M.set_stream(torch.cuda.current_stream().cuda_stream)
        first.fill_(float("nan"))
        if busy:
            z.add_(1.0)
        M.mv_device_f32(dx.data_ptr(), first.data_ptr())
        M.mv_device_f32(dx.data_ptr(), later.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(first, later)
        assert np.all(np.abs(first.cpu().numpy().astype(np.float64) - want) <= bound)
