"""fsi_mpm_substep against the phases called one by one.  The particles sit three
cells apart, so each node has one contributor and both give the same bits; 1,000 of
them take the launch with one warp per CTA, 27,000 the other.  The grid starts with
values of an earlier use, which the call has to clear."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_axis", [1, 10, 30])
def test_substep_equals_its_phases(per_axis):
    import torch

    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    G, rng = 96, np.random.default_rng(2)
    x = 3.6 + 3.0 * np.stack(np.meshgrid(*[np.arange(per_axis)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(x)
    x = ((x + rng.uniform(0, 0.8, (n, 3))) / G).astype(np.float32)
    vol = np.full(n, (1.0 / G) ** 3 / 8, np.float32)
    v = (0.05 * rng.standard_normal((n, 3))).astype(np.float32)

    def solid():
        s = MPMSolid3D(MPMConfig(n_grid=G, dx=1.0 / G, dt=1e-4), n)
        s.init_from_numpy(x, vol, vol * np.float32(1.2), v_np=v)
        for t in (s.t_gv, s.t_gm, s.t_gf):
            t.fill_(0.3)
        return s

    a, b = solid(), solid()
    for _ in range(3):
        a.substep()
        b.clear_grid()
        b.p2g()
        b.grid_update()
        b.g2p()
    for name in ("t_x", "t_v", "t_C", "t_F", "t_Jp", "t_gv", "t_gm", "t_gf"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
