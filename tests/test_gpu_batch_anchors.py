"""The w-correction's factor formed anew every eight planes (planes_in_flight 1 or 2, and
servers): FP32 steps of 64 planes leave the image 7e-7 off under one recurrence, 2.6e-7
with the groups; planes without data, groups without data and FP64 against the oracle."""
import numpy as np
import pytest

import rick_b200 as R
from _util import TOL_FP64, gpu_rows, rel_l2
from test_gpu_sparse_fft import _oracle_image

pytestmark = pytest.mark.gpu


def _case(nx, ny, nw, planes, n=3000):
    rng = np.random.default_rng(nx + ny + nw)
    host = (rng.random(n) * 0.999, rng.random(n) * 0.999 * min(1.0, ny / nx),
            (np.asarray(planes)[rng.integers(0, len(planes), n)] + 0.5) / nw,
            rng.uniform(0.5, 1.5, 2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32))
    res, wmin, wmax = 1.0 / (2.4 * max(nx, ny)), -900.0, 800.0
    want = np.concatenate(_oracle_image(host, nx, ny, nw, "kaiser_bessel", 7, 1, 2, res, wmin,
                                        wmax))
    return host, (res, wmin, wmax), want


def _job(rows, n, nx, ny, nw, precision, meta):
    import torch
    img = torch.full((2, nx * ny), float("nan"), dtype=torch.float64, device="cuda")
    return R.Job(R.Geometry(nx, ny, nw, 7, "kaiser_bessel", precision), n, 1, 2, rows, *meta,
                 img[0], img[1], R.ROWS_ALL), img


def _errors(host, meta, want, nx, ny, nw, precision):
    """Of a batch with planes_in_flight 0, 1 and 2, and of a server."""
    import torch
    rows, n, err = gpu_rows(*host), len(host[0]), []
    for pif in (0, 1, 2):
        job, img = _job(rows, n, nx, ny, nw, precision, meta)
        tune = {"max_chunk": 1024, "grid_blocks_per_sm": 4, "planes_in_flight": pif}
        with R.Batch([job], precision, device=0, tuning=tune) as b:
            b.run(stream=torch.cuda.current_stream())
            torch.cuda.synchronize()
        err.append(rel_l2(img.cpu().numpy(), want))
    job, img = _job(rows, n, nx, ny, nw, precision, meta)
    with R.Server(precision, device=0, hbm_budget=8 * 10**9) as server:
        server.wait(server.submit(job))
    err.append(rel_l2(img.cpu().numpy(), want))
    return err


@pytest.mark.parametrize("nx,ny", [(64, 1024), (64, 2048), (128, 4096)])
def test_many_planes_mixed(nx, ny):
    nw = 64
    host, meta, want = _case(nx, ny, nw, range(nw))
    one, *grouped = _errors(host, meta, want, nx, ny, nw, "mixed")
    for e in grouped:
        assert e < 0.6 * one, (one, grouped)


@pytest.mark.parametrize("nx,ny", [(64, 64), (64, 512), (64, 1024), (64, 4096)])
@pytest.mark.parametrize("nw,planes", [(9, range(9)), (40, [3, 4, 11, 12, 27, 39]), (40, [20]),
                                       (17, [0, 16]), (33, range(2, 33))])
def test_groups(nx, ny, nw, planes):
    host, meta, want = _case(nx, ny, nw, list(planes), 500)
    for precision, tol in (("fp64", TOL_FP64), ("mixed", 1e-6)):
        for e in _errors(host, meta, want, nx, ny, nw, precision):
            assert e < tol, precision
