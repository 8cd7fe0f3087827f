"""The launch variant of a lattice that nobody has timed: the L2 prefetch from
populations larger than the cache in rows of whole 32-cell blocks, the fourth CTA
for FP16 storage or open faces above 200,000 cells, three CTAs otherwise."""

import pytest

from mpm_lbm_b200._lib import FSI_TUNE_LBM_OCC3 as OCC3
from mpm_lbm_b200._lib import FSI_TUNE_LBM_OCC3_PF as PF
from mpm_lbm_b200._lib import FSI_TUNE_LBM_OCC4 as OCC4
from mpm_lbm_b200.lbm import default_tune


@pytest.mark.parametrize("cells,nx,fp16,open_faces,variant", [
    (32 ** 3, 32, False, False, OCC3), (200_000, 100, True, True, OCC3), (200_001, 99, True, False, OCC4),
    (200_001, 99, False, True, OCC4), (200_001, 99, False, False, OCC3), (1_657_888, 32, False, False, OCC3),
    (1_657_920, 32, False, False, PF), (1_657_920, 33, False, False, OCC3), (1_657_920, 33, False, True, OCC4),
    (1_657_920, 32, True, False, OCC4), (3_315_808, 64, True, True, PF), (3_315_808, 63, True, True, OCC4)])
def test_variant_by_size(cells, nx, fp16, open_faces, variant):
    assert default_tune(cells, nx, fp16, open_faces) == variant
