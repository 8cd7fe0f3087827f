"""The binned MPM substeps at the sizes where their chunk kernel changes path:
one particle and partly filled warps, chunks whose node box takes four, two or
one copy of the scatter tile or none (the direct path), many particles in one
cell, and stencils that leave the grid at its upper faces.  Compared with the CPU
oracle after three substeps.

Tolerance: a node sums at most K terms in FP32 in another order than the oracle,
so momenta and masses differ by at most K 2^-24 of the sum of magnitudes; the
affine matrix multiplies a velocity difference by 4 / dx times an offset below
1.5 dx with weights that sum to one, 6 / dx |v| (6 x 32 x 0.9 against max |C| of
6: a factor 30)."""

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

G = 32
DX = 1.0 / G


def _cloud(kind, rng):
    """(positions in cells, bounds on the nodes of some chunk's box, particles a node can see).  The clouds that want
    large boxes fill 48 of the grid's 64 bins, so that no chunk is cut into parts."""
    if kind == "one":
        return np.array([[12.3, 14.6, 9.1]]), (27, 27), 1
    if kind == "warp_and_one":  # 33 particles in two cells
        return 12.6 + rng.uniform(0, 0.9, (33, 3)) + np.array([[1.0, 0, 0]]) * (np.arange(33)[:, None] % 2), (27, 243), 33
    if kind == "one_cell":  # 300 particles in one base cell: three chunks, runs of a whole warp
        return 12.55 + rng.uniform(0, 0.9, (300, 3)), (27, 27), 300
    if kind == "corners":  # stencils that leave the grid at the upper faces (clamped at 1 - dx), and the lower corner
        return np.concatenate([30.4 + rng.uniform(0, 0.6, (40, 3)), 1.0 + rng.uniform(0, 0.6, (20, 3))]), (8, 243), 60
    # base nodes 0 .. k - 1 of every bin: (k + 2)^3 nodes
    cells, per_bin, bounds = {"two_copies": (5, 110, (244, 486)), "one_copy": (7, 90, (487, 972)),
                              "no_tile": (8, 60, (973, 1331))}[kind]
    bins = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:48]
    x = rng.uniform(0, cells - 0.02, (48, per_bin, 3))
    x[:, 0], x[:, 1] = 0.01, cells - 0.03  # both ends of the range in every bin
    return np.clip((0.51 + x + 8.0 * bins[:, None]).reshape(-1, 3), 1.0, 31.0), bounds, per_bin


@pytest.mark.parametrize("kind", ["one", "warp_and_one", "one_cell", "two_copies", "one_copy", "no_tile", "corners"])
@pytest.mark.parametrize("react", [False, True])
def test_chunk_shapes_match_oracle(kind, react):
    from mpm_lbm_b200.config import LBMConfig, MPMConfig, UnifiedSimConfig
    from mpm_lbm_b200.coupling import PenaltyFSICoupler3D
    from mpm_lbm_b200.lbm import LBMFluid3D
    from mpm_lbm_b200.mpm import MPMSolid3D

    rng = np.random.default_rng(7)
    xc, (lo, hi), terms = _cloud(kind, rng)
    x = (xc * DX).astype(np.float32)
    n = len(x)
    vol = np.full(n, DX ** 3 / 8, np.float32)
    mass = vol * np.float32(1.1)
    v = (0.3 * rng.standard_normal((n, 3))).astype(np.float32)
    dt, young, nu = 1.0e-4, 400.0, 0.2
    gpu = MPMSolid3D(MPMConfig(n_grid=G, dx=DX, dt=dt, gravity=(0.0, -9.8, 0.0), young_modulus=young, poisson_ratio=nu,
                               p_rho=1.1, bound=1), n)
    gpu.init_from_numpy(x, vol, mass, v_np=v)
    ora = orc.OracleMPM(G, DX, dt, n, gravity=(0.0, -9.8, 0.0), p_rho=1.1, young_modulus=young, poisson_ratio=nu, bound=1)
    ora.init_from_numpy(x, vol, mass, v_np=v)
    F = (np.eye(3) + 0.05 * rng.standard_normal((n, 3, 3))).astype(np.float32)
    C = (2.0 * rng.standard_normal((n, 3, 3))).astype(np.float32)
    for f, a in ((gpu.F, F), (gpu.C, C)):
        f.from_numpy(a)
    ora.F[...], ora.C[...] = F, C
    cpl = lbm = oc = olbm = None
    if react:
        sim = UnifiedSimConfig(n_grid=G, mpm_dt=dt, lbm_dt_phys_override_s=1.0e-3)
        hydro = (1e-6 * rng.standard_normal((G, G, G, 3))).astype(np.float32)
        lbm = LBMFluid3D(LBMConfig(nx=G, ny=G, nz=G))
        lbm.init_geo_array(np.zeros((G, G, G), np.int8))
        lbm.init_simulation()
        lbm.hydro_force.from_numpy(hydro)
        cpl = PenaltyFSICoupler3D(sim)
        olbm = orc.OracleLBM(G, G, G)
        olbm.hydro_force[...] = hydro
        oc = orc.OracleCoupling(G, sim.dx_norm, sim.lbm_dt_phys)
    gpu.substeps_binned(3, cpl, lbm)
    for _ in range(3):
        ora.clear_grid()
        ora.p2g()
        if react:
            oc.reaction(0, ora, olbm)
        ora.grid_update()
        ora.g2p()
    # the third substep scattered into buffer 2
    box = gpu._bins["t"]["box"][2, : int(gpu._bins["t"]["meta"][3])].cpu().numpy().astype(np.int64)
    nodes = np.prod(np.maximum(box[:, 3:] - box[:, :3] + 1, 0), axis=1)
    assert ((lo <= nodes) & (nodes <= hi)).any(), f"the chunks have {sorted(set(nodes.tolist()))} nodes"
    sums = terms * 2.0 ** -24
    for name, rel in (("x", 1e-6), ("v", max(2e-5, 3 * sums)), ("C", max(2e-5, 30 * 3 * sums)),
                      ("F", max(2e-5, 3 * sums)), ("Jp", max(2e-5, 3 * sums))):
        a, b = getattr(gpu, name).to_numpy(), getattr(ora, name)
        assert np.abs(a - b).max() <= rel * np.abs(b).max(), name
    for name in ("grid_m", "grid_f_ext"):
        a, b = getattr(gpu, name).to_numpy(), getattr(ora, name)
        assert np.abs(a - b).max() <= max(2e-5, sums) * max(np.abs(b).max(), 1e-30), name
