"""Workloads the framework's speed is measured on, through its public entry points.

A case is a plain dict; ``prepare`` builds what a program holds before the call (a driver with its step graph, a
batch, a fluid or a solid object), ``run`` is one pass, ``work`` the bytes and operations the pass cannot do without,
and ``exact`` the same outputs in 64 bits from plain torch (the solver restated below, sharing nothing with the
package but the initial particle positions).

Kinds:
  duct   one FSI step of a duct with a cantilevered plate: FSIDriver3D, moving boundary, S LBM and M MPM substeps
  box    one FSI step of a walled box with a moving elastic body: FSIDriver3D, one LBM step and M MPM substeps
  batch  one batched FSI step of many boxes of uneven size: FSIBatch
  fluid  LBM steps of a channel around a sphere: LBMFluid3D
  solid  MPM substeps of a vibrating block: MPMSolid3D
"""

import math

import numpy as np
import torch

DT = 1.0e-3  # physical seconds per LBM step, as the package's duct and box cases take it
RHO_S = 1.2  # solid density
NU_S = 0.3   # Poisson ratio


# --------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest coupled run (a 32^3 box with a free block, 4,096 particles), stepped call by call as the driver
        # does by default: launches and host calls count
        dict(name="box_32_moving", kind="box", nx=32, ny=32, nz=32, solid="block", cells=8, mode="moving_boundary",
             tau=0.6, e=0.05, m=10, storage="fp32", graph=False),
        # a ragged box with a clamped plate and penalty coupling, its step replayed as a CUDA graph
        dict(name="box_75x52x61_penalty", kind="box", nx=75, ny=52, nz=61, solid="plate", cells=15, mode="penalty",
             tau=0.67, e=0.03, m=10, storage="fp32", graph=True),
        # the benchmarked configuration: 128 x 64 x 64, 24,576 particles, 120 LBM + 40 MPM substeps per FSI step
        dict(name="duct_128", kind="duct", nx=128, ny=64, nz=64, pt=2, ph=32, pw=48, tau=0.55, u=0.05, s=120, m=40,
             transfer="engineering", storage="fp32", graph=True),
        # a smaller ragged duct with the link-area transfer and few substeps, stepped call by call
        dict(name="duct_100_ragged", kind="duct", nx=100, ny=45, nz=39, pt=3, ph=19, pw=25, tau=0.6, u=0.04, s=30,
             m=10, transfer="link_area_experimental", storage="fp32", graph=False),
        # the large duct (196,608 particles, a lattice larger than the L2 cache), in both population storages
        dict(name="duct_256", kind="duct", nx=256, ny=128, nz=128, pt=4, ph=64, pw=96, tau=0.52, u=0.04, s=120, m=40,
             transfer="engineering", storage="fp32", graph=True),
        dict(name="duct_256_fp16", kind="duct", nx=256, ny=128, nz=128, pt=4, ph=64, pw=96, tau=0.52, u=0.04, s=120,
             m=40, transfer="engineering", storage="fp16", graph=True),
        # the batching form: boxes of uneven edges (32-96), modes, stiffness and body sizes advanced together
        dict(name="batch_16", kind="batch", cases=16, m=10, storage="fp32"),
        # one step of a small channel: the smallest call
        dict(name="fluid_32", kind="fluid", nx=32, ny=32, nz=32, steps=1, tau=0.6, open=False, collision="mrt",
             storage="fp32"),
        # ten steps of a ragged open channel, regularized faces, half-precision populations
        dict(name="fluid_150x70x51_open", kind="fluid", nx=150, ny=70, nz=51, steps=10, tau=0.55, open=True,
             collision="mrt", storage="fp16"),
        # ten steps of a large periodic channel with the BGK operator
        dict(name="fluid_192_bgk", kind="fluid", nx=192, ny=176, nz=160, steps=10, tau=0.7, open=False,
             collision="bgk", storage="fp32"),
        # a small block through the reference's own per-phase substep
        dict(name="solid_4k_substep", kind="solid", grid=48, particles=4096, substeps=4, path="substep"),
        # a large body: 1,000,000 particles on a 128^3 grid
        dict(name="solid_1m", kind="solid", grid=128, particles=1000000, substeps=4, path="binned"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "duct", "duct", "duct", "batch", "fluid", "fluid", "solid"])
    storage = rng.choice(["fp32", "fp32", "fp16"])
    if kind == "box":
        nx, ny, nz = (rng.randint(28, 96) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, solid=rng.choice(["block", "plate"]),
                    cells=rng.randint(4, min(16, ny - 8, nz - 8)), mode=rng.choice(["moving_boundary", "penalty"]),
                    tau=round(rng.uniform(0.53, 0.8), 4), e=round(rng.uniform(0.01, 0.1), 4), m=rng.choice([5, 10, 20]),
                    storage=storage, graph=rng.random() < 0.6)
    if kind == "duct":
        nx = _log_int(rng, 64, 224)
        while nx % 32 in (1, 2):  # open faces take no such lattice
            nx += 1
        ny, nz = (_log_int(rng, 30, min(112, nx)) for _ in range(2))  # the unit box's edge is nx cells
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, pt=rng.randint(2, 4), ph=int(ny * rng.uniform(0.35, 0.55)),
                    pw=int(nz * rng.uniform(0.4, 0.75)), tau=round(rng.uniform(0.53, 0.65), 4),
                    u=round(rng.uniform(0.02, 0.05), 4), s=_log_int(rng, 6, 120), m=rng.choice([10, 20, 40]),
                    transfer=rng.choice(["engineering", "engineering", "link_area_experimental"]), storage=storage,
                    graph=rng.random() < 0.7)
    if kind == "batch":
        return dict(kind=kind, cases=rng.randint(2, 16), m=rng.choice([5, 10]), storage=storage)
    if kind == "fluid":
        opened = rng.random() < 0.5
        nx = _log_int(rng, 24, 256)
        while opened and nx % 32 in (1, 2):
            nx += 1
        return dict(kind=kind, nx=nx, ny=_log_int(rng, 24, 160), nz=_log_int(rng, 24, 160), steps=rng.randint(1, 12),
                    tau=round(rng.uniform(0.53, 0.9), 4), open=opened, collision=rng.choice(["mrt", "mrt", "bgk"]),
                    storage=storage)
    grid = rng.choice([32, 40, 64, 96, 128])
    return dict(kind=kind, grid=grid, particles=_log_int(rng, 2000, 3 * (grid // 3) ** 3), substeps=rng.randint(1, 8),
                path=rng.choice(["binned", "binned", "substep"]))


# ------------------------------------------------------------------------------------------------ the package's side
def _rng(seed, salt=0):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _duct_case(c, seed):
    from mpm_lbm_b200.cases import DuctPlateCase

    # the link-area transfer is an option of the driver's configuration
    extra = {} if c["transfer"] == "engineering" else {"reaction_transfer_mode": c["transfer"]}
    u = c["u"] * float(_rng(seed).uniform(0.95, 1.05))
    return DuctPlateCase(lattice=(c["nx"], c["ny"], c["nz"]), tau=c["tau"], u_in=u, plate=(c["pt"], c["ph"], c["pw"]),
                         lbm_substeps=c["s"], mpm_substeps=c["m"], seed=int(seed) & 0x7FFFFFFF, extra=extra)


def _box_case(c, seed):
    from mpm_lbm_b200.batch import BoxCase

    return BoxCase(lattice=(c["nx"], c["ny"], c["nz"]), tau=c["tau"], mode=c["mode"], solid=c["solid"],
                   solid_cells=c["cells"], e_lu=c["e"], mpm_substeps=c["m"], seed=int(seed) & 0x7FFFFFFF)


def _batch_cases(c, seed):
    from mpm_lbm_b200.batch import sample_box_cases

    # the same sizes for every seed (they are the case), other positions and velocities
    boxes = sample_box_cases(c["cases"], seed=3, mpm_substeps=c["m"])
    return [dict(kind="box", nx=b.lattice[0], ny=b.lattice[1], nz=b.lattice[2], solid=b.solid, cells=b.solid_cells,
                 mode=b.mode, tau=b.tau, e=b.e_lu, m=c["m"], storage=c["storage"], graph=False)
            for b in boxes], [int(seed) + 7919 * i for i in range(len(boxes))]


def _body_velocity(c, seed):
    """Initial velocity of a box case's body in normalised units: 0.01 lattice units, seeded direction."""
    d = _rng(seed, 1).normal(size=3)
    return d / np.linalg.norm(d) * 0.01 * (1.0 / max(c["nx"], c["ny"], c["nz"])) / DT


def _box_driver(c, seed):
    drv = _box_case(c, seed).make_driver(storage=c["storage"])
    drv.solid.set_uniform_velocity(*_body_velocity(c, seed))
    drv.use_cuda_graph = bool(c["graph"])
    return drv


def _fluid_arrays(c, seed):
    """Mask, inlet velocity, initial velocity and populations of a fluid case (host, reference order)."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    r = _rng(seed)
    solid = np.zeros((nx, ny, nz), np.int8)
    solid[:, 0, :] = solid[:, -1, :] = solid[:, :, 0] = solid[:, :, -1] = 1
    x, y, z = (np.arange(n, dtype=np.float32) for n in (nx, ny, nz))
    rad = min(0.14 * min(ny, nz), 0.2 * nx)
    cen = (0.4 * nx, 0.5 * ny + r.uniform(-2, 2), 0.5 * nz + r.uniform(-2, 2))
    solid[((x[:, None, None] - cen[0]) ** 2 + (y[None, :, None] - cen[1]) ** 2 + (z[None, None, :] - cen[2]) ** 2)
          < rad * rad] = 1
    u_in = 0.04 * float(r.uniform(0.9, 1.1))
    ph = r.uniform(0, 2 * np.pi, 3)
    prof = (np.sin(np.pi * y / (ny - 1))[:, None] * np.sin(np.pi * z / (nz - 1))[None, :]).astype(np.float32)
    v = np.zeros((nx, ny, nz, 3), np.float32)
    v[..., 0] = u_in * (prof[None] + 0.1 * np.sin(2 * np.pi * x / nx + ph[0])[:, None, None])
    v[..., 1] = 0.1 * u_in * np.sin(4 * np.pi * x / nx + ph[1])[:, None, None] * prof[None]
    v[..., 2] = 0.1 * u_in * np.cos(2 * np.pi * x / nx + ph[2])[:, None, None] * prof[None]
    v[solid > 0] = 0.0
    return solid, (u_in, 0.0, 0.0), v


def _fluid(c, seed):
    from mpm_lbm_b200.config import LBMConfig
    from mpm_lbm_b200.lbm import LBMFluid3D

    solid, u_in, v = _fluid_arrays(c, seed)
    kw = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], niu=(c["tau"] - 0.5) / 3.0,
              relaxation_semantics="standard_lattice_kinematic_viscosity", collision=c["collision"],
              population_storage=c["storage"])
    if c["open"]:
        kw.update(bc_x_left=2, bc_x_right=1, vel_bc_x_left=u_in, rho_bc_x_right=1.0,
                  open_boundary_semantics="regularized_velocity_pressure")
    lbm = LBMFluid3D(LBMConfig(**kw))
    lbm.init_geo_array(solid)
    lbm.init_simulation()
    if not c["open"]:
        lbm.set_force((1.0e-5, 0.0, 0.0))
    pop = _equilibrium(torch.ones(solid.shape, dtype=torch.float64, device="cuda"),
                       torch.as_tensor(v, device="cuda").double().permute(3, 0, 1, 2))
    lbm.F.from_numpy(pop.permute(1, 2, 3, 0).float().contiguous().cpu().numpy())
    lbm.v.from_numpy(v)
    return lbm


def _solid_arrays(c, seed):
    """Jittered block filling the middle of the box at about eight particles per cell, vibrating."""
    n, g = c["particles"], c["grid"]
    r = _rng(seed)
    edge = min(0.6 * g, max(3.0, (n / 8.0) ** (1.0 / 3.0))) / g
    k = math.ceil(n ** (1.0 / 3.0))
    i = np.arange(n)
    idx = np.stack([i % k, (i // k) % k, i // (k * k)], 1)
    x = 0.5 - edge / 2 + edge * (idx + 0.5 + r.uniform(-0.3, 0.3, (n, 3))) / k
    ph = r.uniform(0, 2 * np.pi, 3)
    v = 0.3 * np.stack([np.sin(2 * np.pi * (x[:, (a + 1) % 3] - 0.5) / edge + ph[a]) for a in range(3)], 1)
    vol = np.full(n, edge ** 3 * n / k ** 3 / n, np.float32)
    return x.astype(np.float32), v.astype(np.float32), vol, vol * np.float32(RHO_S)


def _solid_numbers(c):
    """Time step and Young's modulus of a solid case: a wave crosses a tenth of a cell per substep."""
    dt = 2.0e-4 * 64.0 / c["grid"]
    return dt, 400.0


def _solid(c, seed):
    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    x, v, vol, mass = _solid_arrays(c, seed)
    dt, young = _solid_numbers(c)
    s = MPMSolid3D(MPMConfig(n_grid=c["grid"], dx=1.0 / c["grid"], dt=dt, gravity=(0.0, 0.0, 0.0), p_rho=RHO_S,
                             young_modulus=young, poisson_ratio=NU_S), c["particles"])
    s.init_from_numpy(x, vol, mass, v_np=v)
    return s


def prepare(case, seed):
    c = dict(case)
    state = {"case": c}
    if c["kind"] == "duct":
        drv = _duct_case(c, seed).make_driver(storage=c["storage"], graph=bool(c["graph"]))
        if c["graph"]:
            drv.step_once()  # the driver's first step runs eagerly
            drv.autotune()
        _capture(drv, c)
        state["drv"] = drv
    elif c["kind"] == "box":
        drv = _box_driver(c, seed)
        if c["graph"]:
            drv.step_once()
        _capture(drv, c)
        state["drv"] = drv
    elif c["kind"] == "batch":
        from mpm_lbm_b200.batch import FSIBatch

        boxes, seeds = _batch_cases(c, seed)
        batch = FSIBatch(capacity=len(boxes), storage=c["storage"], mpm_substeps=c["m"])
        state["drivers"] = [_box_driver(b, s) for b, s in zip(boxes, seeds)]
        for drv in state["drivers"]:
            batch.add(drv)
        batch.step(use_graph=True)  # captures the batched step
        state["batch"] = batch
    elif c["kind"] == "fluid":
        state["lbm"] = _fluid(c, seed)
    else:
        state["solid"] = _solid(c, seed)
    return state


def _period(c):
    """FSI steps of one pass: the captured graph of a step with an odd number of LBM steps holds two."""
    return 2 if c["graph"] and c.get("s", 1) % 2 else 1


def _capture(drv, c):
    """After a graph-stepped driver's first step: on to a step that replays its graph."""
    if c["graph"]:
        for _ in range(3 if _period(c) == 2 else 1):
            drv.step_once()


def _particles(s):
    return {"x": s.x.to_torch(), "v": s.v.to_torch(), "C": s.C.to_torch(), "F": s.F.to_torch()}


def run(state):
    c = state["case"]
    if c["kind"] in ("duct", "box"):
        drv = state["drv"]
        for _ in range(_period(c)):
            drv.step_once()
        return {"populations": drv.lbm.F.to_torch(), **_particles(drv.solid)}
    if c["kind"] == "batch":
        state["batch"].step(use_graph=True)
        # the batch's cases stay on the device between steps: their state buffers
        return [{"populations": d.lbm.t_pop, "x": d.solid.x.to_torch(), "v": d.solid.v.to_torch(),
                 "F": d.solid.F.to_torch()} for d in state["drivers"]]
    if c["kind"] == "fluid":
        lbm = state["lbm"]
        for _ in range(c["steps"]):
            lbm.step()
        return {"populations": lbm.F.to_torch(), "v": lbm.v.to_torch()}
    s = state["solid"]
    if c["path"] == "binned":
        s.substeps_binned(c["substeps"])
    else:
        for _ in range(c["substeps"]):
            s.substep()
    return _particles(s)


# -------------------------------------------------------------------------------------------------------------- work
# operations of one lattice cell's step (moments, relaxation, reconstruction with opposite directions paired) and of
# one particle's substep (two 27-node transfers of four to seven values, the rotation and the stress)
CELL_FLOPS, PARTICLE_FLOPS, STATE_BYTES = 330.0, 2200.0, 24 * 4


def _coupled_work(c):
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "duct":
        n, steps = 8 * c["pt"] * c["ph"] * c["pw"], c["s"]
    else:
        lo, hi = _box_case(c, 0)._box()
        n, steps = 8 * (hi[0] - lo[0]) * (hi[1] - lo[1]) * (hi[2] - lo[2]), 1
    size = 2 if c["storage"] == "fp16" else 4
    # the populations and the particle state in and out once, the populations read out as 32-bit values
    out = 0 if c.get("batched") else 19 * 4
    period = _period(c)
    return {"bytes": float(cells * (2 * 19 * size + out) + n * 2 * STATE_BYTES),
            "flops": float(period * (cells * steps * CELL_FLOPS + n * c["m"] * PARTICLE_FLOPS))}


def work(case):
    c = dict(case)
    if c["kind"] in ("duct", "box"):
        return _coupled_work(c)
    if c["kind"] == "batch":
        parts = [_coupled_work(dict(b, batched=True)) for b in _batch_cases(c, 0)[0]]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if c["kind"] == "fluid":
        cells = c["nx"] * c["ny"] * c["nz"]
        size = 2 if c["storage"] == "fp16" else 4
        return {"bytes": float(cells * (2 * 19 * size + 22 * 4)), "flops": float(cells * c["steps"] * CELL_FLOPS)}
    return {"bytes": float(c["particles"] * 2 * STATE_BYTES),
            "flops": float(c["particles"] * c["substeps"] * PARTICLE_FLOPS)}


# ------------------------------------------------------------------------------------- the solver in 64 bits (torch)
E = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
     (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
     (0, -1, 1)]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17]


def _moment_rows():
    """The 19 moments of the operator: density, energy, energy square, momenta and heat fluxes, stresses, and the
    third-order moments, as polynomials of the lattice velocities."""
    e = np.array(E, dtype=np.float64)
    x, y, z = e.T
    q = (e * e).sum(1)
    flux = np.select([q == 1, q == 2], [-2.0, 1.0], 0.0)
    diag = (q == 2).astype(np.float64)
    rows = [np.ones(19), q - 1 + 0 * x, np.select([q == 0, q == 1], [1.0, -2.0], 1.0), x, flux * x, y, flux * y, z,
            flux * z, 3 * x * x - q, (3 * x * x - q) * np.where(q == 1, -1.0, 1.0), y * y - z * z,
            (y * y - z * z) * np.where(q == 1, -1.0, 1.0), x * y, y * z, x * z, diag * x * (y * y - z * z),
            diag * y * (z * z - x * x), diag * z * (x * x - y * y)]
    return np.array(rows)


def _equilibrium(rho, u):
    uu = (u * u).sum(0)
    out = []
    for s in range(19):
        eu = E[s][0] * u[0] + E[s][1] * u[1] + E[s][2] * u[2]
        out.append(W[s] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu))
    return torch.stack(out)


class _ExactFluid:
    def __init__(self, shape, tau, solid, collision="mrt", force=(0.0, 0.0, 0.0), inlet=None, regularized=False):
        d = dict(dtype=torch.float64, device="cuda")
        self.static = torch.as_tensor(solid, device="cuda") > 0
        self.solid = self.static.clone()
        self.rho, self.u = torch.ones(shape, **d), torch.zeros((3,) + tuple(shape), **d)
        self.F = _equilibrium(self.rho, self.u)
        self.cf, self.svel = torch.zeros_like(self.u), torch.zeros_like(self.u)
        self.force = torch.tensor(force, **d).reshape(3, 1, 1, 1)
        self.inlet, self.regularized = inlet, regularized
        sv = 1.0 / tau
        so = sv if collision == "bgk" else 8.0 * (2.0 - sv) / (8.0 - sv)
        S = np.array([0, sv, sv, 0, so, 0, so, 0, so] + [sv] * 7 + [so] * 3)
        M = _moment_rows()
        Mi = np.linalg.inv(M)
        self.relax = torch.tensor(Mi @ (S[:, None] * M), **d)
        self.eqm = torch.tensor((Mi * S)[:, [1, 9, 11, 13, 14, 15]], **d)
        self.guo = torch.tensor(Mi @ ((1 - 0.5 * S)[:, None] * M), **d)
        self.impulse_x = None

    def step(self, moving=False):
        """Collide with the stored density and velocity, stream, apply the faces, update the macroscopic fields;
        returns the link force on every solid cell when moving."""
        F, u, rho, shape = self.F, self.u, self.rho, self.F.shape
        eq = torch.stack([(u * u).sum(0), 2 * u[0] ** 2 - u[1] ** 2 - u[2] ** 2, u[1] ** 2 - u[2] ** 2, u[0] * u[1],
                          u[1] * u[2], u[0] * u[2]])
        f = (F.reshape(19, -1) - self.relax @ F.reshape(19, -1) + self.eqm @ eq.reshape(6, -1)).reshape(shape)
        A = self.force + self.cf
        if bool((A != 0).any()):
            uA = (u * A).sum(0)
            g = torch.stack([W[s] * ((sum(E[s][a] * A[a] for a in range(3)) - uA) / 3.0
                                     + sum(E[s][a] * u[a] for a in range(3)) * sum(E[s][a] * A[a] for a in range(3))
                                     / 9.0) for s in range(19)])
            f += (self.guo @ g.reshape(19, -1)).reshape(shape)
        hydro = torch.zeros_like(u) if moving else None
        impulse = torch.zeros(19, dtype=torch.float64, device="cuda")
        new = F.clone()
        for s in range(19):
            o, e = OPP[s], E[s]
            back = tuple(-a for a in e)
            ahead_solid = torch.roll(self.solid, back, (0, 1, 2)) & ~self.solid  # fluid cells whose neighbour is solid
            moved = torch.roll(f[s], e, (0, 1, 2))
            came_from = torch.roll(self.solid, e, (0, 1, 2))
            new[s] = torch.where(~self.solid & ~came_from, moved, new[s])
            if s == 0:
                continue
            bounced = f[s]
            if moving:
                uw = torch.roll(self.svel, back, (1, 2, 3))
                bounced = f[s] - 6.0 * W[s] * rho * (e[0] * uw[0] + e[1] * uw[1] + e[2] * uw[2])
                push = torch.where(ahead_solid, f[s] + bounced, torch.zeros_like(bounced))
                impulse[s] = -e[0] * push.sum()
                push = torch.roll(push, e, (0, 1, 2))
                for a in range(3):
                    if e[a]:
                        hydro[a] += e[a] * push
            new[o] = torch.where(ahead_solid, bounced, new[o])
        self.impulse_x = impulse
        if self.inlet is not None:
            self._faces(new, u, rho)
        self.F = new
        self._macro(u, rho)
        return hydro

    def _faces(self, F, u, rho):
        one = torch.ones_like(rho[0])
        for x, n in ((0, 1), (-1, -2)):
            if self.regularized:
                if x == 0:
                    target = _equilibrium(rho[n], torch.stack([one * v for v in self.inlet]))
                else:
                    target = _equilibrium(one, u[:, n])
                val = target + F[:, n] - _equilibrium(rho[n], u[:, n])
                dirs = [s for s in range(19) if E[s][0] == (1 if x == 0 else -1)]
            else:
                val = _equilibrium(one, torch.stack([one * v for v in self.inlet]) if x == 0 else u[:, n])
                dirs = range(19)
            for s in dirs:
                F[s, x] = torch.where(self.solid[x], F[s, x], val[s])

    def _macro(self, u, rho):
        r = self.F.sum(0)
        j = torch.stack([sum(E[s][a] * self.F[s] for s in range(19) if E[s][a]) for a in range(3)])
        v = (j + 0.5 * (self.force + self.cf)) / r
        self.rho = torch.where(self.solid, torch.ones_like(r), r)
        self.u = torch.where(self.solid, torch.zeros_like(v), v)

    def update_mask(self, phi, threshold=0.5):
        new = self.static | (phi >= threshold)
        freed = self.solid & ~new
        self.solid = new
        self.u = torch.where(freed, self.svel, self.u)
        self.rho = torch.where(freed, torch.ones_like(self.rho), self.rho)
        self.F = torch.where(freed, _equilibrium(self.rho, self.u), self.F)


class _ExactSolid:
    def __init__(self, grid, dt, x, v, vol, mass, young, fixed=None, bound=3):
        t = lambda a: torch.as_tensor(np.asarray(a), device="cuda").double()  # noqa: E731
        self.g, self.dt, self.dx, self.bound = grid, dt, 1.0 / grid, bound
        self.x, self.v, self.vol, self.mass = t(x), t(v), t(vol), t(mass)
        n = len(self.vol)
        self.C = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
        self.eye = torch.eye(3, dtype=torch.float64, device="cuda")
        self.F = self.eye.repeat(n, 1, 1)
        self.fixed = torch.zeros(n, dtype=torch.bool, device="cuda") if fixed is None else \
            torch.as_tensor(np.asarray(fixed), device="cuda") > 0
        self.x0 = self.x.clone()
        self.v[self.fixed] = 0.0
        self.mu = young / (2.0 * (1.0 + NU_S))
        self.la = young * NU_S / ((1.0 + NU_S) * (1.0 - 2.0 * NU_S))

    def stencil(self, shape):
        """(offset, weight, flat node, inside) of the 27 B-spline nodes of every particle on a lattice of `shape`."""
        xp = self.x / self.dx
        base = (xp - 0.5).trunc().long()
        fx = xp - base
        w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2])
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    o = torch.tensor([i, j, k], device="cuda")
                    node = base + o
                    ok = ((node >= 0) & (node < torch.tensor(shape, device="cuda"))).all(1)
                    flat = (node[:, 0] * shape[1] + node[:, 1]) * shape[2] + node[:, 2]
                    wt = w[i, :, 0] * w[j, :, 1] * w[k, :, 2]
                    yield (o - fx) * self.dx, torch.where(ok, wt, torch.zeros_like(wt)), torch.where(ok, flat, 0 * flat)

    def det(self):
        return torch.linalg.det(self.F)

    def substep(self, react=None):
        g, n3 = self.g, self.g ** 3
        R = self.F.clone()
        for _ in range(12):  # Newton's iteration for the orthogonal factor
            R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
        J = self.det()
        P = 2.0 * self.mu * (self.F - R) + (self.la * (J - 1.0) * J)[:, None, None] * \
            torch.linalg.inv(self.F).transpose(1, 2)
        aff = -(self.dt * self.vol / self.dx ** 2)[:, None, None] * (P @ self.F.transpose(1, 2)) + \
            self.mass[:, None, None] * self.C
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
        mom, m, fe = z(n3, 3), z(n3), z(n3, 3)
        pf = react(self) if react is not None else None
        for dpos, w, node in self.stencil((g, g, g)):
            mom.index_add_(0, node, w[:, None] * (self.mass[:, None] * self.v + (aff @ dpos[:, :, None])[:, :, 0]))
            m.index_add_(0, node, w * self.mass)
            if pf is not None:
                fe.index_add_(0, node, w[:, None] * pf)
        live = (m > 0)[:, None]
        gv = torch.where(live, (mom + self.dt * fe) / torch.where(live, m[:, None], torch.ones_like(m[:, None])), mom)
        gv = gv.reshape(g, g, g, 3)
        i = torch.arange(g, device="cuda")
        for a in range(3):
            at = i.reshape([g if b == a else 1 for b in range(3)])
            va = gv[..., a]
            gv[..., a] = torch.where(((at < self.bound) & (va < 0)) | ((at > g - self.bound) & (va > 0)),
                                     torch.zeros_like(va), va)
        gv = gv.reshape(n3, 3)
        v, C = torch.zeros_like(self.v), torch.zeros_like(self.C)
        for dpos, w, node in self.stencil((g, g, g)):
            wv = w[:, None] * gv[node]
            v += wv
            C += 4.0 / self.dx ** 2 * wv[:, :, None] * dpos[:, None, :]
        x = self.x + self.dt * v
        lo, hi = self.dx, 1.0 - self.dx
        v = torch.where((x < lo) & (v < 0) | (x > hi) & (v > 0), torch.zeros_like(v), v)
        x = x.clamp(lo, hi)
        F = (self.eye + self.dt * C) @ self.F
        fix = self.fixed
        self.x = torch.where(fix[:, None], self.x0, x)
        self.v = torch.where(fix[:, None], torch.zeros_like(v), v)
        self.C = torch.where(fix[:, None, None], torch.zeros_like(C), C)
        self.F = torch.where(fix[:, None, None], self.eye, F)


class _ExactCoupled:
    """The coupled step: project the particles, step the fluid, transfer the reaction during the MPM substeps."""

    def __init__(self, fluid, solid, shape, mode, cap, subcycles, m, link_area=False):
        self.fluid, self.solid, self.shape = fluid, solid, shape
        self.mode, self.cap, self.s, self.m, self.link_area = mode, cap, subcycles, m, link_area
        self.steps = subcycles or 1

    def step(self):
        fl, so, n = self.fluid, self.solid, self.shape[0] * self.shape[1] * self.shape[2]
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
        phi, mass, mom = z(n), z(n), z(n, 3)
        vol = so.vol * so.det().clamp(min=0.0) / so.dx ** 3
        for _, w, node in so.stencil(self.shape):
            phi.index_add_(0, node, w * vol)
            mass.index_add_(0, node, w * so.mass)
            mom.index_add_(0, node, (w * so.mass)[:, None] * so.v * (DT / so.dx))
        has = mass > 1.0e-12
        sv = torch.where(has[:, None], mom / torch.where(has, mass, torch.ones_like(mass))[:, None], torch.zeros_like(mom))
        fl.svel = sv.t().reshape((3,) + self.shape).contiguous()
        phi = phi.clamp(0.0, 1.0).reshape(self.shape)
        if self.mode == "penalty":
            on = ~fl.solid & (phi > 1.0e-6)
            f = torch.where(on, 1.0e-3 * phi * fl.rho * (fl.svel - fl.u), torch.zeros_like(fl.u))
            nrm = f.norm(dim=0)
            fl.cf = torch.where(nrm > 1.0e-4, f * (1.0e-4 / nrm), f)
            fl.step()
            hydro = -fl.cf
        else:
            fl.update_mask(phi)
            hydro = 0.0
            for _ in range(self.steps):
                hydro = hydro + fl.step(moving=True)
            hydro = hydro / self.steps
        scale = 1.0
        if self.link_area:  # weights 1 / length of the link, from the last step's force on the solid by direction
            fx = -fl.impulse_x
            wl = torch.tensor([0.0] + [1.0] * 6 + [1.0 / math.sqrt(2.0)] * 12, dtype=torch.float64, device="cuda")
            scale = float(((wl * fx).sum().abs() / (fx.sum().abs() + 1.0e-12)).clamp(0.25, 2.0))
        h, ph = hydro.reshape(3, -1).t().contiguous(), phi.reshape(-1)

        def react(s):
            hs, ps = torch.zeros_like(s.x), torch.zeros_like(s.vol)
            for _, w, node in s.stencil(self.shape):
                hs += w[:, None] * h[node]
                ps += w * ph[node]
            pf = hs * (s.dx / DT ** 2) * (s.vol * s.det().clamp(min=0.0))[:, None]
            if self.mode == "penalty":
                return pf
            pf = pf * scale
            nrm = pf.norm(dim=1, keepdim=True)
            pf = torch.where(nrm > self.cap, pf * (self.cap / nrm), pf)
            return torch.where((ps > 1.0e-6)[:, None], pf, torch.zeros_like(pf))

        for _ in range(self.m):
            so.substep(react)

    def outputs(self):
        return {"populations": self.fluid.F.permute(1, 2, 3, 0), **_exact_particles(self.solid)}


def _exact_particles(s):
    return {"x": s.x, "v": s.v, "C": s.C, "F": s.F}


def _exact_duct(c, seed):
    case = _duct_case(c, seed)
    solid, parts = case.geometry()
    shape = (c["nx"], c["ny"], c["nz"])
    fluid = _ExactFluid(shape, c["tau"], solid, inlet=(case.u_in, 0.0, 0.0))
    dx = 1.0 / c["nx"]
    so = _ExactSolid(c["nx"], c["s"] * DT / c["m"], parts["x"], np.zeros_like(parts["x"]), parts["vol0"], parts["mass"],
                     case.e_lu * (dx / DT) ** 2, parts["fixed"])
    return _ExactCoupled(fluid, so, shape, "moving_boundary", case.reaction_cap, c["s"], c["m"],
                         link_area=c["transfer"] != "engineering")


def _exact_box(c, seed):
    case = _box_case(c, seed)
    solid, parts = case.geometry()
    shape = (c["nx"], c["ny"], c["nz"])
    n = max(shape)
    fluid = _ExactFluid(shape, c["tau"], solid, force=case.body_force)
    v = np.tile(_body_velocity(c, seed).astype(np.float32), (len(parts["x"]), 1))
    so = _ExactSolid(n, DT / c["m"], parts["x"], v, parts["vol0"], parts["mass"], c["e"] * ((1.0 / n) / DT) ** 2,
                     parts["fixed"])
    return _ExactCoupled(fluid, so, shape, c["mode"], 1.0e-8 * (128.0 / n) ** 3, 0, c["m"])


def exact(case, seed):
    c = dict(case)
    if c["kind"] in ("duct", "box"):
        sim = _exact_duct(c, seed) if c["kind"] == "duct" else _exact_box(c, seed)
        for _ in range(3 * _period(c) if c["graph"] else 1):  # the steps of prepare(), and run()'s
            sim.step()
        return sim.outputs()
    if c["kind"] == "batch":
        out = []
        for b, s in zip(*_batch_cases(c, seed)):
            sim = _exact_box(b, s)
            for _ in range(2):
                sim.step()
            p = _exact_particles(sim.solid)
            out.append({"populations": None, "x": p["x"], "v": p["v"], "F": p["F"]})
        return out
    if c["kind"] == "fluid":
        solid, u_in, v = _fluid_arrays(c, seed)
        fl = _ExactFluid(solid.shape, c["tau"], solid, collision=c["collision"],
                         force=(0.0, 0.0, 0.0) if c["open"] else (1.0e-5, 0.0, 0.0),
                         inlet=u_in if c["open"] else None, regularized=True)
        fl.u = torch.as_tensor(v, device="cuda").double().permute(3, 0, 1, 2)
        fl.F = _equilibrium(fl.rho, fl.u)
        for _ in range(c["steps"]):
            fl.step()
        return {"populations": fl.F.permute(1, 2, 3, 0), "v": fl.u.permute(1, 2, 3, 0)}
    x, v, vol, mass = _solid_arrays(c, seed)
    dt, young = _solid_numbers(c)
    so = _ExactSolid(c["grid"], dt, x, v, vol, mass, young)
    for _ in range(c["substeps"]):
        so.substep()
    return _exact_particles(so)
