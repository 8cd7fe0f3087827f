"""Automatic re-binning of a cloud that crosses cells: re-binned every three
substeps, never, and in one call (which is never re-binned inside) it moves alike,
and only the first has other bins afterwards.

Tolerance: with |v| = 15 the gather's 27 terms, rounded once each, put a velocity off
by up to 27 x 2^-24 x 15 = 2.4e-5 and the affine matrix by 6 / dx times that, 0.014:
per substep 2.4e-9 in a position, which is itself rounded to 6e-8, and 1.4e-6 in F;
over 18 substeps 1.1e-6 and 2.5e-5."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6000, 3 << 17])
def test_rebinning_of_a_moving_cloud(n):
    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    G, rng = 96, np.random.default_rng(7)
    side = np.arange(76)
    x = 20.0 + 0.5 * np.stack(np.meshgrid(side, side, side, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = ((x + rng.uniform(0, 0.5, x.shape)) / G).astype(np.float32)
    vol = np.full(n, (0.5 / G) ** 3, np.float32)
    v = np.tile(np.float32([15.0, -10.0, 12.0]), (n, 1))  # 0.14 cells per substep
    x_of, f_of, chunks = [], [], []
    for interval, calls in ((3, [1] * 18), (10 ** 9, [1] * 18), (3, [18])):
        s = MPMSolid3D(MPMConfig(n_grid=G, dx=1.0 / G, dt=1e-4), n)
        s.init_from_numpy(x, vol, vol * np.float32(1.2), v_np=v)
        s.rebin_interval = interval
        for c in calls:
            s.substeps_binned(c)
        x_of.append(s.x.to_numpy())
        f_of.append(s.F.to_numpy())
        chunks.append(s._bins["t"]["chunk"][: int(s._bins["t"]["meta"][0])].cpu().numpy())
    assert np.abs(x_of[0] - x).max() * G > 2  # several cells
    for k in (1, 2):
        np.testing.assert_allclose(x_of[0], x_of[k], rtol=0, atol=2e-6)
        np.testing.assert_allclose(f_of[0], f_of[k], rtol=0, atol=5e-5)
    assert np.array_equal(chunks[1], chunks[2])
    assert chunks[0].shape != chunks[1].shape or not np.array_equal(chunks[0], chunks[1])
