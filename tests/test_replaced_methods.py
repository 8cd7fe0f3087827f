"""A subclass or wrapper of the methods that one fused library call stands for is
still reached: MPMSolid3D.substep runs the four phases, a subcycled FSI step every
substep of the lattice, when one of them is replaced.  The library's calls are
recorded, not made."""

import types

import pytest

from mpm_lbm_b200 import lbm as lbm_module
from mpm_lbm_b200 import mpm as mpm_module
from mpm_lbm_b200.config import LBMConfig, MPMConfig
from mpm_lbm_b200.driver import FSIDriver3D

PHASES = ["fsi_mpm_p2g", "fsi_mpm_grid_update", "fsi_mpm_g2p"]


@pytest.fixture
def calls(monkeypatch):
    names = []
    for module in (lbm_module, mpm_module):
        monkeypatch.setattr(module, "call", lambda name, *args: names.append(name))
        monkeypatch.setattr(module, "stream_handle", lambda: None)
    return names


def _solid(cls=mpm_module.MPMSolid3D):
    return cls(MPMConfig(n_grid=8, dx=0.125, dt=1e-4), 8, device="cpu")


@pytest.mark.parametrize("name", ["clear_grid", "p2g", "grid_update", "g2p"])
@pytest.mark.parametrize("how", ["subclass", "instance", "class"])
def test_replaced_phase_is_reached(calls, monkeypatch, name, how):
    own = getattr(mpm_module.MPMSolid3D, name)
    seen = []

    def wrapper(self):
        seen.append(name)
        own(self)

    if how == "subclass":
        s = _solid(type("Solid", (mpm_module.MPMSolid3D,), {name: wrapper}))
    else:
        s = _solid()
        if how == "instance":
            setattr(s, name, types.MethodType(wrapper, s))
        else:
            monkeypatch.setattr(mpm_module.MPMSolid3D, name, wrapper)
    s.substep()
    s.substep()
    assert seen == [name] * 2 and calls == PHASES * 2


def test_own_phases_go_in_one_call(calls):
    _solid().substep()
    assert calls == ["fsi_mpm_substep"]


def _subcycled(cls, substeps):
    lbm = cls(LBMConfig(nx=8, ny=8, nz=8), device="cpu")
    lbm.tau_f = 0.6
    nothing = lambda *a: None  # noqa: E731
    drv = types.SimpleNamespace(lbm=lbm, total_lbm_substeps=0, _project=nothing, _t=nothing,
                                _advance_mpm_with_moving_boundary_reaction=nothing,
                                config=types.SimpleNamespace(lbm_substeps_per_fsi_step=substeps,
                                                             dynamic_solid_threshold=0.5))
    FSIDriver3D._step_moving_boundary_subcycled(drv)
    assert drv.total_lbm_substeps == lbm.steps == lbm._sample_count == substeps
    assert lbm._old_equals_solid == (substeps > 1) and lbm.dirstats_enabled
    return lbm


@pytest.mark.parametrize("substeps", [1, 2, 5])
@pytest.mark.parametrize("name,times", [("step_moving_bounceback", 0), ("accumulate_moving_boundary_force_sample", 0),
                                        ("reinitialize_new_fluid_cells", 0), ("mark_repeat_mask_update", 1)])
def test_replaced_substep_method_is_reached(calls, name, times, substeps):
    own = getattr(lbm_module.LBMFluid3D, name)
    seen = []

    def wrapper(self):
        seen.append((self.steps, self.dirstats_enabled))
        own(self)

    _subcycled(type("Fluid", (lbm_module.LBMFluid3D,), {name: wrapper}), substeps)
    assert len(seen) == substeps - times and calls.count("fsi_lbm_substep") == substeps
    if name == "step_moving_bounceback":
        assert seen == [(s, s == substeps - 1) for s in range(substeps)]


@pytest.mark.parametrize("substeps", [1, 2, 5])
def test_own_substeps_go_in_one_call(calls, substeps):
    _subcycled(lbm_module.LBMFluid3D, substeps)
    assert calls.count("fsi_lbm_substeps") == (substeps > 1) and calls.count("fsi_lbm_substep") == 1


def test_substeps_that_end_in_an_error_leave_the_statistics_on(calls):
    class Fluid(lbm_module.LBMFluid3D):
        def step_moving_bounceback(self):
            raise ValueError("stop")

    lbm = Fluid(LBMConfig(nx=8, ny=8, nz=8), device="cpu")
    lbm.tau_f = 0.6
    with pytest.raises(ValueError, match="stop"):
        lbm.step_moving_bounceback_run(2)
    assert lbm.dirstats_enabled
