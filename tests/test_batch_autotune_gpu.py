"""The autotuner tries a digit width only where the batch's sort has one."""
import pytest

import nexusbvh_gb300 as nxb
from tests import stages as S
from tests.test_batch_gpu import make_batch

pytestmark = pytest.mark.gpu

PER_WIDTH = 2 * 3 * 3  # H-PLOC grids, fusion points, block sizes


@pytest.mark.parametrize("counts,widths", [([900, 0, 4000, 33], 1),               # a cluster per mesh
                                           ([70_000, 30_000], 1),                 # passes within every mesh
                                           ([65_537] + [5] * 80, 5),              # passes over mesh and code
                                           ([3000] + [2] * 3000, 4)])             # 4-bit digits would take 11 passes
def test_candidates(gpu, counts, widths):
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.sort_digit_bits = 7
    batch.set_tuning(t)
    chosen = batch.autotune(S.dev(make_batch(counts, seed=2)), repeats=1)
    assert chosen.candidates_tried == PER_WIDTH * widths
    if widths == 1:
        assert chosen.sort_digit_bits == 7
