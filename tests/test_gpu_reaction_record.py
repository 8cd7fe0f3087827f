"""The reaction record of a sequence of binned substeps is the last substep's, and
the other two are zero: M substeps in one call against M - 1 and one more.

Tolerance: the particle positions of the two runs differ by the order of the grid's
atomic sums, 1e-6 of a cell's fields per substep; the record's sums run over a few
hundred particles of one sign."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 7])
def test_record_is_the_last_substeps(M):
    from mpm_lbm_b200.cases import DuctPlateCase

    drv = DuctPlateCase(lattice=(40, 20, 18), plate=(2, 8, 8), lbm_substeps=3, mpm_substeps=2).make_driver()
    for _ in range(3):
        drv.step_once()
    coupler, solid = drv.mb_coupler, drv.solid
    snap = solid.snapshot()
    records = []
    for parts in ([M], [M - 1, 1]):
        solid.restore(snap)
        for m in parts:
            solid.substeps_binned(m, coupler, drv.lbm)
        records.append(coupler._reaction_stats())
        for slot in set(range(3)) - {coupler._binned_slot}:
            r = coupler.binned_stats.read(slot)
            assert r.active_reaction_particle_count == 0 and not any(r.net_particle_reaction)
            assert not any(r.net_grid_reaction) and r.max_particle_reaction_norm == r.max_grid_reaction_norm == 0.0
    a, b = records
    assert a.active_reaction_particle_count == b.active_reaction_particle_count > 0
    for name in ("net_particle_reaction", "net_grid_reaction"):
        x, y = np.array(getattr(a, name)[:]), np.array(getattr(b, name)[:])
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max() > 0
    for name in ("max_particle_reaction_norm", "max_grid_reaction_norm"):
        assert abs(getattr(a, name) - getattr(b, name)) <= 1e-5 * getattr(b, name)
