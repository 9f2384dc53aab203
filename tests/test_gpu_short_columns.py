"""A batch of one job whose columns are short and few: the mixed form, which works through
two columns a thread where FP64 has one, took 1.7 times as long as FP64 (279 us against
168 for 64^2 x 64 planes) while its column loop was too long for the instruction cache;
0.95 times with the steps of planes without data in a loop of their own."""
import numpy as np
import pytest

import rick_b200 as R
from _util import TOL_FP64, TOL_MIXED, gpu_rows, rel_l2
from test_gpu_sparse_fft import _oracle_image

pytestmark = pytest.mark.gpu


def _rows(nx, n, nw, planes):
    rng = np.random.default_rng(nx + n)
    uu, vv = (np.clip(0.5 + 0.1 * rng.standard_normal(n), 0, 0.999) for _ in range(2))
    ww = (np.asarray(planes)[rng.integers(0, len(planes), n)] + 0.5) / nw
    return (uu, vv, ww, rng.uniform(0.5, 1.5, 2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32))


def _batch(rows, n, nx, nw, precision, res, wmin, wmax):
    import torch
    img = torch.empty(2, nx * nx, dtype=torch.float64, device="cuda")
    job = R.Job(R.Geometry(nx, nx, nw, 7, "kaiser_bessel", precision), n, 1, 2, rows, res, wmin,
                wmax, img[0], img[1], R.ROWS_ALL)
    tune = {"max_chunk": 2048, "grid_blocks_per_sm": 6, "planes_in_flight": 0}
    return R.Batch([job], precision, device=0, tuning=tune), img


def test_mixed_takes_no_longer_than_fp64():
    import torch
    nx, nw, n = 64, 64, 20000
    rows = gpu_rows(*_rows(nx, n, nw, range(nw)))
    us = {}
    for precision in ("fp64", "mixed"):
        batch, _ = _batch(rows, n, nx, nw, precision, 1 / 200, -90.0, 80.0)
        t = []
        with batch:
            for _ in range(15):
                e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                e0.record()
                batch.run(stream=torch.cuda.current_stream())
                e1.record()
                torch.cuda.synchronize()
                t.append(e0.elapsed_time(e1))
        us[precision] = sorted(t)[len(t) // 2]
    assert us["mixed"] < 1.3 * us["fp64"], us


@pytest.mark.parametrize("nx", [64, 512, 1024])
@pytest.mark.parametrize("planes", [[0, 7], [3, 4, 11], [11]])
def test_planes_without_data(nx, planes):
    """Gaps of one to six planes between those with data, in both forms."""
    import torch
    nw, n = 12, 500
    host = _rows(nx, n, nw, planes)
    res, wmin, wmax = 1.0 / (2.4 * nx), -310.0, 290.0
    want = np.concatenate(_oracle_image(host, nx, nx, nw, "kaiser_bessel", 7, 1, 2, res, wmin,
                                        wmax))
    rows = gpu_rows(*host)
    for precision, tol in (("fp64", TOL_FP64), ("mixed", TOL_MIXED)):
        batch, img = _batch(rows, n, nx, nw, precision, res, wmin, wmax)
        with batch:
            batch.run(stream=torch.cuda.current_stream())
            torch.cuda.synchronize()
        assert rel_l2(img.cpu().numpy(), want) < tol, precision
