"""Batches whose jobs share a class of a stage: several jobs of one column length that
take the finishing kernel (1024 and 2048 rows, uneven widths and planes, a job without
rows between them), and rows of every sample schedule of the batch (fewer than 8, 8 to
15, 16 to 31 and more loads of four, two and one samples)."""
import numpy as np
import pytest

import rick_b200 as R
from _util import TOL_FP64, TOL_MIXED, gpu_rows, rel_l2
from test_gpu_sparse_fft import _oracle_image

pytestmark = pytest.mark.gpu


def _run(jobs, precision):
    """jobs: (nx, ny, nw, nchan, npol, rows); every image against the oracle's."""
    import torch
    batch, host, images = [], [], []
    for k, (nx, ny, nw, nchan, npol, n) in enumerate(jobs):
        rng = np.random.default_rng(k + n)
        nv = nchan * npol
        h = (np.clip(0.5 + 0.1 * rng.standard_normal(n), 0, 0.999),
             np.clip(0.5 + 0.1 * rng.standard_normal(n), 0, 0.999) * min(1.0, ny / nx),
             rng.random(n) * 0.999, rng.uniform(0.5, 1.5, npol * n).astype(np.float32),
             rng.standard_normal(nv * n).astype(np.float32),
             rng.standard_normal(nv * n).astype(np.float32))
        rows = gpu_rows(*h) if n else tuple(torch.empty(1, device="cuda") for _ in range(6))
        img = torch.full((2, nx * ny), float("nan"), dtype=torch.float64, device="cuda")
        batch.append(R.Job(R.Geometry(nx, ny, nw, 7, "gauss", precision), n, nchan, npol, rows,
                           1.0 / (2.4 * max(nx, ny)), -300.0 - k, 290.0, img[0], img[1], R.ROWS_ALL))
        host.append(h)
        images.append(img)
    tune = {"max_chunk": 1024, "grid_blocks_per_sm": 4, "planes_in_flight": 0}
    with R.Batch(batch, precision, device=0, tuning=tune) as b:
        b.run(stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
    for k, (nx, ny, nw, nchan, npol, n) in enumerate(jobs):
        got = images[k].cpu().numpy().ravel()
        if n == 0:
            assert not got.any(), k
            continue
        want = np.concatenate(_oracle_image(host[k], nx, ny, nw, "gauss", 7, nchan, npol,
                                            1.0 / (2.4 * max(nx, ny)), -300.0 - k, 290.0))
        assert rel_l2(got, want) < (TOL_FP64 if precision == "fp64" else TOL_MIXED), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_finish_of_several_jobs(precision):
    _run([(64, 1024, 3, 1, 2, 700), (128, 2048, 2, 1, 2, 500), (256, 1024, 5, 1, 2, 0),
          (512, 1024, 2, 1, 2, 900), (64, 2048, 6, 1, 2, 800), (64, 2048, 1, 1, 2, 0),
          (192 + 64, 1024, 1, 1, 2, 600), (256, 2048, 4, 1, 2, 1000)], precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rows", [33, 1000])
def test_sample_schedules(precision, rows):
    _run([(64, 64, 2, nchan, npol, rows + k) for k, (nchan, npol) in enumerate(
        [(1, 2), (7, 4), (8, 4), (15, 4), (16, 4), (31, 4), (32, 4), (48, 4), (9, 2), (17, 2),
         (35, 2), (9, 1), (17, 1), (33, 1), (12, 3)])], precision)
