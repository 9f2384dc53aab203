"""Every transform length of the row and the column pass (64..8192, two and three
radix passes, last radices 2..16, the two halves at 8192) against the oracle, in
both forms, at row counts that leave a pair of the mixed form half empty."""
import numpy as np
import pytest

import rick_b200 as R
from _util import TOL_FP64, TOL_MIXED, gpu_image, gpu_rows, rel_l2
from test_gpu_sparse_fft import _oracle_image

pytestmark = pytest.mark.gpu

LENGTHS = [64, 128, 256, 512, 1024, 2048, 4096, 8192]


def _case(nx, ny, nw, n, planes, seed):
    rng = np.random.default_rng(seed)
    uu = rng.uniform(0.0, 1.0, n)
    vv = rng.uniform(0.0, min(1.0, ny / nx) * 0.999, n)  # v is scaled by 1/nx as u is
    ww = (np.asarray(planes)[rng.integers(0, len(planes), n)] + rng.uniform(0.1, 0.9, n)) / nw
    return (uu, vv, ww, rng.uniform(0.5, 1.5, 2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32))


@pytest.mark.parametrize("n_rows", [1, 4000])
@pytest.mark.parametrize("nx,ny", [(n, 64) for n in LENGTHS] + [(64, n) for n in LENGTHS[1:]] +
                         [(8192, 128)])
def test_lengths(nx, ny, n_rows):
    nw, planes = 6, [0, 2, 5]
    sup = 7
    if nx < ny:
        planes = [1, 2]  # neighbouring planes, the first and the last without rows
    host = _case(nx, ny, nw, n_rows, planes, nx + 3 * ny + n_rows)
    rows = gpu_rows(*host)
    res, wmin, wmax = 1.0 / (2.4 * max(nx, ny)), -310.0, 290.0
    want = np.concatenate(_oracle_image(host, nx, ny, nw, "kaiser_bessel", sup, 1, 2, res, wmin,
                                        wmax))
    for precision, tol in (("fp64", TOL_FP64), ("mixed", TOL_MIXED)):
        re, im, st = gpu_image(rows, n_rows, nx, ny, nw, sup, "kaiser_bessel", 1, 2, res, wmin,
                               wmax, selection=R.ROWS_ALL, precision=precision)
        err = rel_l2(np.concatenate([re, im]), want)
        assert err < tol, (precision, err, st["fft_rows"])
