"""The automatic re-binning of large and small clouds: the same motion as without
it.  Tolerances as for the binned substep against the plain one: positions 1e-6,
deformation gradients 1e-5."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3 << 17) - 1, 3 << 17])
def test_rebinning_keeps_the_motion(n):
    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    G, rng = 96, np.random.default_rng(7)
    side = np.arange(76)
    x = 20.0 + 0.5 * np.stack(np.meshgrid(side, side, side, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = ((x + rng.uniform(0, 0.5, x.shape)) / G).astype(np.float32)
    vol = np.full(n, (0.5 / G) ** 3, np.float32)
    v = np.tile(np.float32([0.3, -0.2, 0.25]), (n, 1))
    out = []
    for interval in (None, 10 ** 9):
        s = MPMSolid3D(MPMConfig(n_grid=G, dx=1.0 / G, dt=1e-4), n)
        s.init_from_numpy(x, vol, vol * np.float32(1.2), v_np=v)
        assert s.rebin_interval == (8 if n >= 3 << 17 else 64)
        if interval:
            s.rebin_interval = interval
        for _ in range(18):
            s.substeps_binned(1)
        out.append((s.x.to_numpy(), s.F.to_numpy()))
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=0, atol=1e-6)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-5)
