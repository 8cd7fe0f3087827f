"""The first binned substep of a solid that has already run one-phase substeps: the
grid they left behind is not part of it (momentum and mass would count twice).
Tolerances as for the binned substep against the plain one: positions 1e-6,
deformation gradients 1e-5, grid masses 1e-5 of the largest."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rebin_first", [False, True])
@pytest.mark.parametrize("before", ["substep", "phases", "grid_write"])
def test_binned_after_one_phase(before, rebin_first):
    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    G, rng = 32, np.random.default_rng(5)
    x = (8.0 + rng.uniform(0, 8, (4000, 3))) / G
    vol = np.full(len(x), 0.125 / G ** 3, np.float32)
    v = (0.2 * rng.standard_normal(x.shape)).astype(np.float32)
    out = []
    for binned in (True, False):
        s = MPMSolid3D(MPMConfig(n_grid=G, dx=1.0 / G, dt=1e-4, young_modulus=100.0, p_rho=1.1), len(x))
        s.init_from_numpy(x.astype(np.float32), vol, vol * np.float32(1.1), v_np=v)
        if before == "grid_write":
            s.grid_m.from_numpy(np.ones((G, G, G), np.float32))
        else:
            for _ in range(2):
                if before == "substep":
                    s.substep()
                else:
                    s.clear_grid()
                    s.p2g()
                    s.grid_update()
                    s.g2p()
        if binned:
            if rebin_first:
                s.rebin()
            s.substeps_binned(2)
        else:
            s.substep()
            s.substep()
        out.append((s.x.to_numpy(), s.F.to_numpy(), s.grid_m.to_numpy()))
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=0, atol=1e-6)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-5)
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=0, atol=1e-5 * out[1][2].max())
