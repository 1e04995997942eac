"""The FP64-equivalent ensemble step with its march blocks first in the grid
(up to two per SM) and spread among the ring blocks (more): every cell within the
form's bound of the FP64 form."""
import pytest

from test_gpu_ensemble_df import REL_L2, run_pair, worst_rel_l2
from test_gpu_ensemble_masks import domain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nx,ny", [
    (1, 4, 5),       # one march block
    (8, 148, 60),    # strips of 8 rows, 80 march blocks
    (19, 118, 126),  # 304: the most that come first
    (20, 118, 126),  # 320
])
def test_march_and_ring_blocks_take_every_cell(gpulib, n, nx, ny):
    doms = [domain(nx, ny, "SNEW"[k % 4], 0.02 * (k % 2), k) for k in range(n)]
    ref, _, got, _ = run_pair(gpulib, doms, 12)
    assert worst_rel_l2(doms, ref, got) <= REL_L2
