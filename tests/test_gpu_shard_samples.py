"""The sample pass of w-plane shards: every schedule (rows of fewer than 8, 8 to 15, 16
to 31 and more loads of four, two and one samples; shards below, at and above half of
the planes) against the oracle, and the time of a shard that keeps half of the rows."""
import numpy as np
import pytest

import oracle as O
import rick_b200 as R
from _util import TOL_FP64, gpu_rows, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan,npol", [(2, 2), (8, 4), (12, 4), (14, 4), (17, 4), (31, 4), (33, 4), (9, 2),
                                        (17, 2), (7, 1), (9, 1), (19, 1), (35, 1)])
@pytest.mark.parametrize("planes", [(0, 3), (2, 4), (1, 7)])
def test_shard_cube(nchan, npol, planes):
    import torch
    nx, nw, n = 64, 8, 2003
    rng = np.random.default_rng(nchan * 10 + npol)
    uu, vv, ww = rng.random(n) * 0.999, rng.random(n) * 0.999, rng.random(n) * 0.999
    vr = rng.standard_normal(n * nchan * npol).astype(np.float32)
    vr[rng.random(vr.size) < 0.01] = np.nan
    host = (uu, vv, ww, rng.uniform(0.5, 1.5, n * npol).astype(np.float32), vr,
            rng.standard_normal(n * nchan * npol).astype(np.float32))
    want, _ = O.wstack("gauss", nw, nchan, npol, uu, vv, ww, vr, host[5], host[3], 1 / nx, 1 / nw,
                       7, nx, nx)
    first, count = planes
    want = want.reshape(nw, -1)[first: first + count]
    geom = R.Geometry(nx, nx, nw, 7, "gauss", "fp64")
    with R.Plan(geom, n, nchan, npol, device=0, planes=planes) as plan:
        plan.grid(n, gpu_rows(*host), R.ROWS_ALL)
        out = torch.empty(2 * count * nx * nx, dtype=torch.float64, device="cuda")
        plan.export_cube(out, dst_is_host=False)
        torch.cuda.synchronize()
        st = plan.stats()
    assert rel_l2(out.cpu().numpy(), want) < TOL_FP64
    kept = int(np.isin((ww * nw).astype(int), np.arange(first, first + count)).sum())
    assert st["rows_gridded"] == kept and st["rows_other_shard"] == n - kept


def test_half_shard_leaves_the_other_half_unread():
    """Rows of 256 samples, the shard holding half of the planes and of the rows: with
    the other half's samples read too its sample pass takes as long as a whole-cube
    plan's (1.01 of it measured), without them 0.66."""
    import torch
    nx, nw, n, nchan, npol = 512, 8, 600_000, 64, 4
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)
    uu, vv, ww = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * 0.999
                  for _ in range(3))
    wt = torch.ones(n * npol, device="cuda")
    vis = torch.rand(n * nchan * npol, generator=gen, device="cuda")
    img = torch.empty(2, nx * nx, dtype=torch.float64, device="cuda")
    ms = {}
    for planes in (None, (0, nw // 2), (nw // 2, nw // 2)):
        with R.Plan(R.Geometry(nx, nx, nw), n, nchan, npol, device=0, planes=planes) as plan:
            plan.set_timing(True)
            t = []
            for _ in range(12):
                plan.image(n, (uu, vv, ww, wt, vis, vis), 1e-4, -50.0, 50.0, img[0], img[1],
                           R.ROWS_ALL)
                torch.cuda.synchronize()
                t.append(plan.stage_ms()["bin_scatter"])
            ms[planes] = sorted(t)[len(t) // 2]
    for planes in ((0, nw // 2), (nw // 2, nw // 2)):
        assert ms[planes] < 0.85 * ms[None], ms


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_shards_of_finished_columns(precision):
    """Columns of 1024 rows, whose sums a finishing kernel turns into the image with the
    factor of a shard's own lowest plane: the shards' images add up to the oracle's."""
    import torch
    from _util import TOL_MIXED
    from test_gpu_sparse_fft import _oracle_image
    nx, nw, n = 1024, 6, 900
    rng = np.random.default_rng(3)
    host = (rng.random(n) * 0.999, rng.random(n) * 0.999, rng.random(n) * 0.999,
            rng.uniform(0.5, 1.5, 2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32),
            rng.standard_normal(2 * n).astype(np.float32))
    res, wmin, wmax = 1.0 / (2.4 * nx), -310.0, 290.0
    want = np.concatenate(_oracle_image(host, nx, nx, nw, "gauss", 7, 1, 2, res, wmin, wmax))
    rows = gpu_rows(*host)
    total = np.zeros(2 * nx * nx)
    for planes in ((0, 2), (2, 3), (5, 1)):
        with R.Plan(R.Geometry(nx, nx, nw, 7, "gauss", precision), n, 1, 2, device=0,
                    planes=planes) as plan:
            img = torch.empty(2, nx * nx, dtype=torch.float64, device="cuda")
            plan.image(n, rows, res, wmin, wmax, img[0], img[1], R.ROWS_ALL)
            torch.cuda.synchronize()
            total += img.cpu().numpy().ravel()
    assert rel_l2(total, want) < (TOL_FP64 if precision == "fp64" else TOL_MIXED)
