"""CSR products over the row lengths and row counts where the lanes per row change, against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows,mean", [(1, 1), (3, 40), (200, 5), (70001, 5), (65537, 11), (33000, 13), (16384, 17),
                                        (16385, 30), (9000, 81), (8193, 251), (4097, 300), (70, 1001), (33, 2100)])
def test_spmv_lanes_per_row(nrows, mean):
    import torch
    import blackwell_kernels as bk

    rng = np.random.default_rng(nrows + mean)
    length = rng.integers(0, 2 * mean + 1, nrows)          # empty rows and rows of twice the mean
    ptr = np.zeros(nrows + 1, dtype=np.int32)
    np.cumsum(length, out=ptr[1:])
    nnz = int(ptr[-1])
    col = rng.integers(0, nrows, nnz).astype(np.int32)
    val = (rng.standard_normal(nnz) + 1j * rng.standard_normal(nnz)).astype(np.complex64)
    x = (rng.standard_normal(nrows) + 1j * rng.standard_normal(nrows)).astype(np.complex64)
    y = (rng.standard_normal(nrows) + 1j * rng.standard_normal(nrows)).astype(np.complex64)
    d = [torch.from_numpy(a).cuda() for a in (ptr, col, val, x, y)]
    bk.spmv_csr(*d, alpha_re=0.5, alpha_im=-1.5, beta_re=2.0, beta_im=0.25)

    prod = val.astype(np.complex128) * x[col].astype(np.complex128)
    mag = np.abs(val.astype(np.complex128)) * np.abs(x[col].astype(np.complex128))
    rows = np.repeat(np.arange(nrows), length)
    dot = np.bincount(rows, prod.real, nrows) + 1j * np.bincount(rows, prod.imag, nrows)
    size = np.bincount(rows, mag, nrows)
    want = (0.5 - 1.5j) * dot + (2.0 + 0.25j) * y
    # the compensated dot is rounded once (and to second order in u per entry);
    # alpha * dot + beta * y adds at most four roundings of its terms
    u = 2.0 ** -24
    tol = 8 * u * (abs(0.5 - 1.5j) * np.abs(dot) + abs(2 + 0.25j) * np.abs(y)) + 4 * (length + 1) * u * u * size
    assert np.all(np.abs(d[4].cpu().numpy() - want) <= tol)
