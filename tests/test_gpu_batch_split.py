"""Batched MPM substeps where the launch cuts the chunks into parts (few cases on
the device) and where it does not (many): the same cases alone, in a batch of one,
next to empty slots and in a batch of twelve end alike.  Tolerances as for the batch
against single runs: positions 1e-6, deformation gradients 1e-5, populations 1e-5."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity,copies", [(1, 1), (5, 1), (12, 12)])
def test_batch_sizes_match_single_runs(capacity, copies):
    import torch

    from mpm_lbm_b200.batch import BoxCase, FSIBatch

    case = BoxCase(lattice=(34, 32, 30), tau=0.6, mode="moving_boundary", solid="block", solid_cells=9, mpm_substeps=5,
                   seed=4)

    def fields(drv):
        return drv.lbm.F.to_numpy(), drv.lbm.solid.to_numpy(), drv.solid.x.to_numpy(), drv.solid.F.to_numpy()

    alone = case.make_driver()
    alone.solid.set_uniform_velocity(0.2, 0.1, -0.1)
    for _ in range(3):
        alone.step_once()
    want = fields(alone)
    batch = FSIBatch(capacity=capacity, mpm_substeps=5)
    for _ in range(copies):
        drv = case.make_driver()
        drv.solid.set_uniform_velocity(0.2, 0.1, -0.1)
        batch.add(drv, slot=None if copies > 1 else capacity - 1)
    for _ in range(3):
        batch.step(use_graph=True)
    torch.cuda.synchronize()
    for slot in range(capacity - copies, capacity):
        got = fields(batch.sync_case(slot))
        np.testing.assert_array_equal(got[1], want[1])
        np.testing.assert_allclose(got[0], want[0], rtol=1e-5, atol=1e-7)
        np.testing.assert_allclose(got[2], want[2], rtol=0, atol=1e-6)
        np.testing.assert_allclose(got[3], want[3], rtol=0, atol=1e-5)
