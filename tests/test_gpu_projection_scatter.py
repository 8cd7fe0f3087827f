"""Edges of both projections' launches.

The ordered projection (fsi_project_ordered) against the oracle, bit for bit:
cells whose number of contributors lies at the sizes where the register sort
changes and where the ids are taken in several passes, and bounding boxes whose
keys end at, before and after the blocks of the scan.

The float-atomic projection (fsi_project, the batched form's) at the edges of
its warp-wide runs: one particle, partly filled warps, particles in memory order
and shuffled, one crowded cell, stencils that leave the lattice.  Compared with
the serial order's sums (fsi_project_ordered): a cell adds at most K terms in
FP32 in another order, each term rounded a few times, so a sum differs by at most
(K + 8) 2^-24 of the cell's sum of magnitudes; the velocities are quotients of two
such sums."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 24


def _cloud(kind, rng):
    if kind == "one":
        return np.array([[7.3, 11.6, 5.2]])
    if kind == "block":  # memory order: eight consecutive particles per cell
        cells = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        return (6.5 + cells + rng.uniform(0.02, 0.98, (64, 8, 3))).reshape(-1, 3)[:483]
    if kind == "shuffled":
        return rng.permutation(_cloud("block", rng))
    if kind == "crowded":
        return 9.55 + rng.uniform(0, 0.9, (161, 3))
    return np.concatenate([rng.uniform(-0.4, 1.0, (33, 3)), rng.uniform(N - 1.0, N + 0.4, (34, 3))])  # edges


@pytest.mark.parametrize("kind", ["one", "block", "shuffled", "crowded", "edges"])
def test_unordered_projection_matches_ordered(kind):
    from mpm_lbm_b200.config import LBMConfig, MPMConfig, UnifiedSimConfig
    from mpm_lbm_b200.coupling import MPMToLBMProjector3D
    from mpm_lbm_b200.lbm import LBMFluid3D
    from mpm_lbm_b200.mpm import MPMSolid3D

    rng = np.random.default_rng(3)
    x = (_cloud(kind, rng) / N).astype(np.float32)
    n = len(x)
    solid = MPMSolid3D(MPMConfig(n_grid=N, dx=1.0 / N, dt=1e-4), n)
    vol = np.full(n, (1.0 / N) ** 3 / 8, np.float32)
    solid.init_from_numpy(x, vol, vol * np.float32(1.2), v_np=rng.uniform(0.2, 1.0, (n, 3)).astype(np.float32))
    sim = UnifiedSimConfig(n_grid=N, mpm_dt=1e-4, lbm_dt_phys_override_s=1.0e-3)
    lbm = LBMFluid3D(LBMConfig(nx=N, ny=N, nz=N))
    proj = MPMToLBMProjector3D(sim)
    proj.project(solid, lbm)
    ref = [t.clone() for t in (lbm.t_phi, lbm.t_smass, lbm.t_svel)]
    want = proj.get_stats()
    proj.project_unordered(solid, lbm)
    rel = (min(n, 216) + 8) * 2.0 ** -24  # at 8 per cell 27 cells see a node; every term is positive
    if kind == "crowded":
        rel = (n + 8) * 2.0 ** -24
    for got, exp, name, k in ((lbm.t_phi, ref[0], "phi", 1), (lbm.t_smass, ref[1], "mass", 1), (lbm.t_svel, ref[2], "vel", 2)):
        d = (got - exp).abs()
        assert bool((d <= k * rel * exp.abs() + 1e-30).all()), (name, float((d / (exp.abs() + 1e-30)).max()), rel)
    got = proj.get_stats()
    assert got["active_cell_count"] == want["active_cell_count"]
    np.testing.assert_allclose(got["projected_mass"], want["projected_mass"], rtol=rel)


def _ordered_cloud(kind, rng):
    if kind == "counts":  # one base cell each, far apart
        counts = (1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 256, 257, 511, 512, 513, 1024, 1025, 1600)
        cells = [(3 + 6 * (i % 3), 3 + 6 * (i // 3 % 3), 3 + 9 * (i // 9)) for i in range(len(counts))]
        x = np.concatenate([np.array(c) + rng.uniform(0.55, 1.45, (m, 3)) for c, m in zip(cells, counts)])
        return rng.permutation(x)
    # keys = 15 * 15 * 18 = 4050, 16 * 16 * 16 = 4096, 17 * 15 * 17 = 4335, 24 ** 3 = 13824
    ext = np.array({"keys_4050": (15, 15, 18), "keys_4096": (16, 16, 16), "keys_4335": (17, 15, 17),
                    "keys_13824": (24, 24, 24)}[kind])
    lo = np.minimum(2, N - ext)
    x = lo + 0.5 + np.floor(rng.uniform(0, 1, (700, 3)) * ext) + rng.uniform(0.05, 0.95, (700, 3))
    return np.concatenate([x, [lo + 0.7], [lo + ext - 0.3]])


@pytest.mark.parametrize("kind", ["counts", "keys_4050", "keys_4096", "keys_4335", "keys_13824"])
def test_ordered_projection_launch_edges(kind):
    from mpm_lbm_b200.config import LBMConfig, MPMConfig, UnifiedSimConfig
    from mpm_lbm_b200.coupling import MPMToLBMProjector3D
    from mpm_lbm_b200.lbm import LBMFluid3D
    from mpm_lbm_b200.mpm import MPMSolid3D
    from oracle import oracle as orc

    rng = np.random.default_rng(5)
    x = (_ordered_cloud(kind, rng) / N).astype(np.float32)
    n = len(x)
    vol = np.full(n, (1.0 / N) ** 3 / 8, np.float32)
    mass = vol * np.float32(1.2)
    v = rng.standard_normal((n, 3)).astype(np.float32)
    sim = UnifiedSimConfig(n_grid=N, mpm_dt=1e-4, lbm_dt_phys_override_s=1.0e-3)
    lbm = LBMFluid3D(LBMConfig(nx=N, ny=N, nz=N))
    solid = MPMSolid3D(MPMConfig(n_grid=N, dx=1.0 / N, dt=1e-4), n)
    solid.init_from_numpy(x, vol, mass, v_np=v)
    ol, om = orc.OracleLBM(N, N, N), orc.OracleMPM(N, 1.0 / N, 1e-4, n)
    om.x[...], om.v[...], om.Jp[...], om.vol0[...], om.mass[...] = x, v, 1.0, vol, mass
    orc.OracleCoupling(N, sim.dx_norm, sim.lbm_dt_phys).project(om, ol)
    proj = MPMToLBMProjector3D(sim)
    for _ in range(2):  # the second call finds the scratch as the first one left it
        proj.project(solid, lbm)
        np.testing.assert_array_equal(lbm.solid_phi.to_numpy(), ol.solid_phi)
        np.testing.assert_array_equal(lbm.solid_mass.to_numpy(), ol.solid_mass)
        np.testing.assert_array_equal(lbm.solid_vel.to_numpy(), ol.solid_vel)
