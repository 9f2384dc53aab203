"""Images whose column pass leaves its sums to the finishing kernel (columns of 1024
points and more, too many of them to deal the planes to several blocks) against the
oracle: every such length, the first planes empty, one plane, and no rows at all."""
import numpy as np
import pytest

import rick_b200 as R
from _util import TOL_FP64, TOL_MIXED, gpu_image, gpu_rows, rel_l2
from test_gpu_fft_lengths import _case
from test_gpu_sparse_fft import _oracle_image

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1024, 1024), (512, 2048), (512, 4096), (512, 8192)])
@pytest.mark.parametrize("nw,planes,n", [(6, [3, 5], 300), (1, [0], 300), (6, [3], 0)])
def test_finish(nx, ny, nw, planes, n):
    host = _case(nx, ny, nw, max(n, 1), planes, nx + ny + nw)
    rows = gpu_rows(*host)
    res, wmin, wmax = 1.0 / (2.4 * max(nx, ny)), -310.0, 290.0
    want = None
    if n:
        want = np.concatenate(_oracle_image(host, nx, ny, nw, "kaiser_bessel", 7, 1, 2, res, wmin,
                                            wmax))
    for precision, tol in (("fp64", TOL_FP64), ("mixed", TOL_MIXED)):
        re, im, _ = gpu_image(rows, n, nx, ny, nw, 7, "kaiser_bessel", 1, 2, res, wmin, wmax,
                              selection=R.ROWS_ALL, precision=precision)
        got = np.concatenate([re, im])
        if n:
            assert rel_l2(got, want) < tol, precision
        else:
            assert not got.any(), precision
