"""Dense tiles, whose records are split over several work items of the gridder: item
sizes at their edges against the oracle, and the parts an FP32 cube's cells add up."""
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


@pytest.mark.parametrize("n,items", [(8000, 125), (10_000, 79), (75_000, 74), (600_000, 147)])
def test_parts_added_into_fp32_cells(n, items):
    """Each item of a tile is added into its cells: in the mixed form, whose cells are
    FP32, at most 128 of fewer than 1024 records, and 256 of more."""
    host = _one_tile(n, 64, 8, 23)
    _, st = gpu_grid(gpu_rows(*host), n, 64, 64, 1, 7, "gauss", 1, 1, "mixed", R.ROWS_ALL)
    assert st["work_items"] == items
