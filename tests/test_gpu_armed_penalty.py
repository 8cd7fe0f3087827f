"""A penalty force that is armed before a moving-boundary step is refused (penalty
steps use static bounce-back, fluid.py:2099-2103) by the run of substeps as by the
single substep, and stays armed."""

import pytest

pytestmark = pytest.mark.gpu


def test_run_of_substeps_refuses_an_armed_penalty():
    from mpm_lbm_b200._lib import FsiError
    from mpm_lbm_b200.cases import DuctPlateCase
    from mpm_lbm_b200.coupling import PenaltyFSICoupler3D

    drv = DuctPlateCase(lattice=(40, 20, 18), plate=(2, 8, 8), lbm_substeps=3, mpm_substeps=2).make_driver()
    drv.step_once()
    lbm = drv.lbm
    penalty = PenaltyFSICoupler3D(drv.sim)
    penalty.clear_force_fields(lbm)
    penalty.build_penalty_force(lbm)
    steps, pop = lbm.steps, lbm.t_pop.clone()
    for refused in (lambda: lbm.step_moving_bounceback_run(2), lbm.step_moving_bounceback, drv.step_once):
        with pytest.raises(FsiError, match="penalty steps use static bounce-back"):
            refused()
        assert lbm.steps == steps and lbm._penalty is not None
    lbm.step()  # the armed force goes into the next static step
    assert lbm.steps == steps + 1 and lbm._penalty is None and not bool((lbm.t_pop == pop).all())
