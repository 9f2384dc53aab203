"""Dense tiles, whose records are split over several work items of the gridder: item
sizes at their edges against the oracle, and the error of an FP32 cube's cells."""
import numpy as np
import pytest

import oracle as O
import rick_b200 as R
from _util import TOL_FP64, TOL_MIXED, gpu_grid, gpu_rows, rel_l2

pytestmark = pytest.mark.gpu


def _one_tile(n, nx, lo, hi):
    """n rows of one sample whose cells are lo to hi on both axes, equal weights."""
    rng = np.random.default_rng(n)
    return [(lo + (hi - lo) * rng.random(n)) / nx, (lo + (hi - lo) * rng.random(n)) / nx,
            np.full(n, 0.5), np.ones(n, np.float32), rng.standard_normal(n).astype(np.float32),
            rng.standard_normal(n).astype(np.float32)]


@pytest.mark.parametrize("n", [63, 64, 65, 1024, 8192, 8193, 16400, 131073, 262145])
@pytest.mark.parametrize("nx", [64, 50])
def test_item_sizes(nx, n):
    """Below and above the sizes at which a tile is split and its items grow."""
    host = _one_tile(n, nx, 4, 27)
    want, _ = O.wstack("kaiser_bessel", 1, 1, 1, host[0], host[1], host[2], host[4], host[5],
                       host[3], 1 / nx, 1.0, 7, nx, nx)
    for precision, tol in (("fp64", TOL_FP64), ("mixed", TOL_MIXED)):
        got, st = gpu_grid(gpu_rows(*host), n, nx, nx, 1, 7, "kaiser_bessel", 1, 1, precision,
                           R.ROWS_ALL)
        assert rel_l2(got, want) < tol
        assert (st["work_items"] > 1) == (n > 64)


@pytest.mark.parametrize("data", ["equal", "noise"])
@pytest.mark.parametrize("n,nx,nw", [(75_000, 64, 1), (75_000, 50, 1), (600_000, 64, 2)])
def test_fp32_cells_of_dense_tiles(data, n, nx, nw):
    """Tiles of more than 64 items are added up in FP64 before they become FP32 cells, so
    a cell's error is what its items' 32-bit sums lose.  Such a sum's unit is below
    2^-29 of the item's bound, sum (|re| + |im|) wmax, so an item of m records of like
    size rounds each contribution by at most 2^-30 * 2 m wmax |s|, evenly distributed: a
    standard deviation of m wmax |s| 2^-29 / sqrt(3).  Against a cell's own root mean
    square of sqrt(records) w_rms |s| (noise; the equal samples' cells are larger) that is
    m 2^-29 / sqrt(3) wmax / w_rms, and with the Gaussian's wmax / w_rms below 6 over its
    seven cells squared: m * 6.5e-9.  FP32 contributions and cells add 2^-24 twice."""
    rng = np.random.default_rng(n)
    host = _one_tile(n, nx, 8, 23)
    host[2] = (rng.integers(0, nw, n) + 0.5) / nw
    if data == "equal":
        host[4] = host[5] = np.ones(n, np.float32)
    cube = {}
    for precision in ("fp64", "mixed"):
        cube[precision], st = gpu_grid(gpu_rows(*host), n, nx, nx, nw, 7, "gauss", 1, 1, precision,
                                       R.ROWS_ALL)
        assert st["work_items"] > 64 * nw
    m = max(64, n // (8 * 148))
    assert rel_l2(cube["mixed"], cube["fp64"]) < 6.5e-9 * m + 2.0 ** -23


def test_wide_sums_start_at_zero_again():
    """Grids of other rows after one with dense tiles, with and without dense tiles."""
    import torch
    nx, n = 64, 75_000
    with R.Plan(R.Geometry(nx, nx, 1, 7, "gauss", "mixed"), n, 1, 1, device=0) as plan:
        for k, m in enumerate((n, 900, n, n)):
            host = _one_tile(m, nx, 8 + k, 20 + k)
            plan.grid(m, gpu_rows(*host), R.ROWS_ALL)
            out = torch.empty(2 * nx * nx, dtype=torch.float64, device="cuda")
            plan.export_cube(out, dst_is_host=False)
            torch.cuda.synchronize()
            want, _ = O.wstack("gauss", 1, 1, 1, host[0], host[1], host[2], host[4], host[5],
                               host[3], 1 / nx, 1.0, 7, nx, nx)
            assert rel_l2(out.cpu().numpy(), want) < TOL_MIXED, k


@pytest.mark.parametrize("grid,nw", [((64, 64), 1), ((64, 96), 3), ((256, 256), 2)])
def test_as_many_wide_tiles_as_there_can_be(grid, nw):
    """Every tile of the grid just above 64 items of 64 records (nothing on tile edges, so
    that a row is one record), or as many as the rows give."""
    nx, ny = grid
    tiles = (nx // 32) * (ny // 32) * nw
    per = 64 * 64 + 1
    rng = np.random.default_rng(tiles)
    n = per * min(tiles, 17)  # items stay at 64 records up to 75,776 rows
    k = np.arange(n) // per
    tx, ty, w = k % (nx // 32), (k // (nx // 32)) % (ny // 32), k // ((nx // 32) * (ny // 32))
    host = [(32 * tx + 5 + 20 * rng.random(n)) / nx, (32 * ty + 5 + 20 * rng.random(n)) / nx,
            (w + 0.5) / nw, np.ones(n, np.float32), rng.standard_normal(n).astype(np.float32),
            rng.standard_normal(n).astype(np.float32)]
    want, _ = O.wstack("kaiser_bessel", nw, 1, 1, host[0], host[1], host[2], host[4], host[5],
                       host[3], 1 / nx, 1 / nw, 7, nx, ny)
    got, st = gpu_grid(gpu_rows(*host), n, nx, ny, nw, 7, "kaiser_bessel", 1, 1, "mixed",
                       R.ROWS_ALL)
    assert st["work_items"] == 65 * min(tiles, 17)
    assert rel_l2(got, want) < 1e-6
