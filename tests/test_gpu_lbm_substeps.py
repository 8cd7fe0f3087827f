"""fsi_lbm_substeps: n moving-boundary substeps in one call leave the state that
n single substeps leave.  The populations and face planes depend on no
floating-point atomic and are compared bit for bit; a link-force sum adds at
most 18 terms per substep in an order that varies, so the accumulator may
differ by 18 n 2^-24 of its largest value."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5])
@pytest.mark.parametrize("storage,boundary", [("fp32", "equilibrium_all_population_reset"),
                                              ("fp16", "regularized_velocity_pressure_limited")])
def test_substeps_equal_single_substeps(n, storage, boundary):
    import torch

    from mpm_lbm_b200.cases import DuctPlateCase

    case = DuctPlateCase(lattice=(40, 20, 18), plate=(2, 8, 8), lbm_substeps=3, mpm_substeps=2, open_boundary=boundary)
    states = []
    for together in (False, True):
        drv = case.make_driver(storage=storage)
        drv.step_once()
        lbm = drv.lbm
        lbm.dirstats_enabled = False
        lbm.clear_moving_boundary_force_accumulator()
        if together:
            lbm.step_moving_bounceback_run(n)
        else:
            for _ in range(n):
                lbm.step_moving_bounceback()
                lbm.accumulate_moving_boundary_force_sample()
        states.append((lbm.t_pop.clone(), lbm.t_plane[:4].clone(), lbm._accum_tensor().clone(),
                       (lbm.parity, lbm.pp, lbm.last_pp, lbm.bc_pending, lbm.steps, lbm._sample_count)))
    assert states[0][3] == states[1][3]
    assert torch.equal(states[0][0], states[1][0]) and torch.equal(states[0][1], states[1][1])
    a, b = states[0][2], states[1][2]
    assert float((a - b).abs().max()) <= 18 * n * 2.0 ** -24 * float(a.abs().max())


def test_substeps_refuse_other_modes():
    import ctypes

    from mpm_lbm_b200._lib import FSI_MODE_DIRSTATS, FSI_MODE_MOVING_BB, last_error, load
    from mpm_lbm_b200.config import LBMConfig
    from mpm_lbm_b200.lbm import LBMFluid3D

    lbm = LBMFluid3D(LBMConfig(nx=8, ny=8, nz=8))
    lbm.init_simulation()
    lib = load()
    for mode in (0, FSI_MODE_MOVING_BB | FSI_MODE_DIRSTATS):
        ctl = lbm._ctl(mode)
        rc = lib.fsi_lbm_substeps(ctypes.byref(lbm.state), ctypes.byref(lbm.params), ctypes.byref(ctl), 2,
                                  lbm._stream())
        assert rc == -1 and "moving-boundary" in last_error()
