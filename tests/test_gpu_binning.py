"""The sample pass over its schedules (one lane a row with block-wise places, four to
32 lanes a row, loads of four, two and one samples) and the bin scan over one and
several blocks: the gridded cube against the oracle's, and every row accounted for."""
import numpy as np
import pytest

import oracle as O
import rick_b200 as R
from _util import TOL_FP64, gpu_grid, gpu_rows, rel_l2

pytestmark = pytest.mark.gpu


def _rows(seed, n, nchan, npol, dense):
    rng = np.random.default_rng(seed)
    if dense:  # most rows in a few bins
        uu, vv = (np.clip(0.5 + 0.01 * rng.standard_normal(n), 0, 0.9999) for _ in range(2))
    else:      # a block's rows in as many bins as there are: places beyond the table
        uu, vv = rng.random(n) * 0.9999, rng.random(n) * 0.9999
    ww = rng.random(n)
    vr = rng.standard_normal(n * nchan * npol).astype(np.float32)
    vr[rng.random(vr.size) < 0.01] = np.nan
    return (uu, vv, ww, rng.uniform(0.5, 1.5, n * npol).astype(np.float32), vr,
            rng.standard_normal(n * nchan * npol).astype(np.float32))


@pytest.mark.parametrize("nchan,npol", [(1, 1), (1, 2), (3, 2), (7, 1), (2, 3), (2, 4), (7, 4),
                                        (8, 4), (15, 1), (12, 4), (17, 4), (33, 4)])
@pytest.mark.parametrize("n", [1, 33, 513, 6001])
def test_sample_schedules(nchan, npol, n):
    nx = 1000 if n == 513 else 1024   # 1/1000 is no power of two: the dividing path
    nw = 2 if n < 6001 else 12        # 2048 bins in one scan block, 12288 in two
    host = _rows(n + nchan, n, nchan, npol, dense=n == 513)
    uu, vv, ww, wt, vr, vi = host
    want, _ = O.wstack("gauss", nw, nchan, npol, uu, vv, ww, vr, vi, wt, 1 / nx, 1 / nw, 7, nx, nx)
    got, st = gpu_grid(gpu_rows(*host), n, nx, nx, nw, 7, "gauss", nchan, npol,
                       selection=R.ROWS_ALL)
    assert rel_l2(got, want) < TOL_FP64
    assert st["rows_gridded"] + st["rows_dropped"] == n and st["rows_dropped"] == 0


@pytest.mark.parametrize("nchan,npol,offset", [(4, 4, 1), (4, 2, 2), (3, 2, 2), (3, 2, 1)])
def test_samples_at_odd_addresses(nchan, npol, offset):
    """Sample arrays that start off a 16-byte (8-byte) boundary take shorter loads."""
    import torch
    nx, nw, n = 512, 4, 2000
    host = _rows(7, n, nchan, npol, dense=False)
    rows = list(gpu_rows(*host))
    for k in (4, 5):
        buf = torch.empty(rows[k].numel() + offset, dtype=torch.float32, device="cuda")
        buf[offset:] = rows[k]
        rows[k] = buf[offset:]
    uu, vv, ww, wt, vr, vi = host
    want, _ = O.wstack("kaiser_bessel", nw, nchan, npol, uu, vv, ww, vr, vi, wt, 1 / nx, 1 / nw, 7,
                       nx, nx)
    got, _ = gpu_grid(rows, n, nx, nx, nw, 7, "kaiser_bessel", nchan, npol, selection=R.ROWS_ALL)
    assert rel_l2(got, want) < TOL_FP64
