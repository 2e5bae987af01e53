"""CSR products with a few rows far above the mean (a star's centre, an arrowhead's first rows): at the length where the
whole warp takes a row, for every number of lanes, against FP64; and no slower than the row by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(rng, length, ncols):
    ptr = np.zeros(len(length) + 1, dtype=np.int32)
    np.cumsum(length, out=ptr[1:])
    nnz = int(ptr[-1])
    col = rng.integers(0, ncols, nnz).astype(np.int32)
    val = (rng.standard_normal(nnz) + 1j * rng.standard_normal(nnz)).astype(np.complex64)
    return ptr, col, val


@pytest.mark.parametrize("nrows,mean,lanes", [(70001, 3, 1), (40003, 12, 2), (17001, 30, 4), (8195, 100, 8), (4099, 300, 16)])
def test_long_rows(nrows, mean, lanes):
    import torch
    import blackwell_kernels as bk

    rng = np.random.default_rng(nrows)
    length = rng.integers(0, 2 * mean + 1, nrows)
    edge = 64 * lanes
    # the first, neighbours in one warp, the last; at the limit and either side, and one of many warps' steps
    for r, n in ((0, edge + 1), (1, edge), (2, edge - 1), (3, edge + 1), (4, 3001), (5, edge + 130), (nrows // 2, 20011),
                 (nrows - 1, edge + 33)):
        length[r] = n
    ptr, col, val = _matrix(rng, length, nrows)
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
    # as the rows of ordinary length: a compensated dot rounded once, then four roundings
    u = 2.0 ** -24
    tol = 8 * u * (abs(0.5 - 1.5j) * np.abs(dot) + abs(2 + 0.25j) * np.abs(y)) + 4 * (length + 1) * u * u * size
    assert np.all(np.abs(d[4].cpu().numpy() - want) <= tol)


def test_star_takes_as_long_as_its_centre():
    import torch
    import blackwell_kernels as bk

    rng = np.random.default_rng(5)
    n = 1 << 17

    def time(length):
        ptr, col, val = _matrix(rng, length, n)
        x = torch.ones(n, dtype=torch.complex64, device="cuda")
        y = torch.zeros(len(length), dtype=torch.complex64, device="cuda")
        d = [torch.from_numpy(a).cuda() for a in (ptr, col, val)]
        best = 1e9
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            bk.spmv_csr(*d, x, y)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    star = np.full(n, 2)
    star[0] = n
    # the one row by itself has a warp; the others are a small part of a launch of that length, and one lane
    # would take some 30 times as long
    assert time(star) <= 3 * time(np.array([n]))
