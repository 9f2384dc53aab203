"""Equal bits: a batch whose work items hold a tile's records whole repeats itself bit
for bit; a plan, which splits tiles and deals planes for speed, to rounding."""
import numpy as np
import pytest

import rick_b200 as R
from _util import gpu_rows, rel_l2

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    uu, vv = (np.clip(0.5 + 0.08 * rng.standard_normal(n), 0, 0.999) for _ in range(2))
    return gpu_rows(uu, vv, rng.random(n) * 0.999, rng.uniform(0.5, 1.5, 2 * n),
                    rng.standard_normal(4 * n), rng.standard_normal(4 * n))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,nw,n,planes_in_flight", [(128, 4, 5400, 0), (64, 17, 3000, 1),
                                                      (1024, 20, 40000, 1), (2048, 3, 60000, 0)])
def test_batch_of_whole_tiles(precision, nx, nw, n, planes_in_flight):
    import torch
    rows = _rows(n, nx)
    img = torch.empty(2, nx * nx, dtype=torch.float64, device="cuda")
    job = R.Job(R.Geometry(nx, nx, nw, 7, "kaiser_bessel", precision), n, 2, 2, rows, 1e-4, -200.0,
                180.0, img[0], img[1], R.ROWS_ALL)
    tune = {"max_chunk": 1 << 20, "grid_blocks_per_sm": 6, "planes_in_flight": planes_in_flight}
    with R.Batch([job], precision, device=0, tuning=tune) as batch:
        first = None
        for _ in range(6):
            img.fill_(float("nan"))
            batch.run(stream=torch.cuda.current_stream())
            torch.cuda.synchronize()
            if first is None:
                first = img.clone()
            assert torch.equal(img, first)
    with R.Plan(job.geom, n, 2, 2, device=0) as plan:
        plan.image(n, rows, 1e-4, -200.0, 180.0, img[0], img[1], R.ROWS_ALL)
        torch.cuda.synchronize()
    assert rel_l2(img.cpu().numpy(), first.cpu().numpy()) < (1e-13 if precision == "fp64" else 2e-6)
