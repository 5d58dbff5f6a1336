"""The work a user of this framework has it do, as cases to time.

Each case goes through the package's public entry points (Solver, Assembly, BatchSolver, the painting
functions, the closure's training functions) with the sizes of the repository's own benchmark
workloads and tests, or generic ones.  A case is a dict of plain values; ``prepare`` makes what a
program holds before the call, ``run`` is one pass, ``exact`` the same pass in 64 bits by plain
torch (no code of the package on its arithmetic), ``work`` what one pass cannot do without.

Kinds:
  run      a time loop (Solver.run) and the macroscopic fields at its end
  loop     a time loop of single calls with link-wise bounce-back and a force reading
  batch    many small 2D channels stepped together (BatchSolver)
  train    one optimiser step of the learned subgrid closure
  outputs  the outputs of one state: density and velocity, Q-criterion, mass and momentum
  setup    a domain painted and initialised on the device
"""
from __future__ import annotations

import ctypes
import math
from pathlib import Path

import numpy as np
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_Grid, LBM_method, _capi, closure, geometry, preprocess, tgv, workloads
from mojo_lbm_gb300.assembly import Assembly
from mojo_lbm_gb300.batch import BatchSolver
from mojo_lbm_gb300.lattice import get_lattice
from mojo_lbm_gb300.solver import Solver

LATTICE = {"D2Q9": 0, "D3Q19": 1, "D3Q27": 2}
CLOSURE_FILE = Path(closure.__file__).parent / "data" / "tgv_re1600_512to256_closure.npz"
DEV = "cuda"
LARGEST = 100 * 256 ** 3  # cell updates of the largest listed time loop


def _run(name, lattice, shape, tile, steps, flow, **kw):
    case = dict(kind="run", lattice=lattice, nx=shape[0], ny=shape[1], nz=shape[2], tile=tile, steps=steps, flow=flow,
                method="db", coll="SRT", les="off", f16=False, arith="exact", tau=0.884, U=0.1)
    case.update(kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # smallest: the reference's cylinder drivers call the step, then the bounce-back of the body, from a
        # host loop and read the force every so often: a small channel, every call its own launches
        dict(name="loop_channel_d2q9", kind="loop", nx=320, ny=128, steps=16, Re=20.0, offset=0.0),
        # the reference's CPU-runnable cavity (256 x 256, a 20,000-step run), taken 1000 steps at a time
        _run("cavity_d2q9_256", "D2Q9", (256, 256, 1), "16,16,1", 1000, "cavity", tau=1.265),
        # the benchmark's default workload: float32 lid-driven cube
        _run("cavity_d3q19_256_fp32", "D3Q19", (256, 256, 256), "8,8,4", 100, "cavity", tau=1.265),
        # the same cube with 16-bit storage, as memory-limited runs take it
        _run("cavity_d3q19_256_f16c", "D3Q19", (256, 256, 256), "8,8,4", 100, "cavity", tau=1.265, f16=True,
             arith="fast"),
        # the high-Reynolds configuration: 27 directions, entropic collision, LES, in-place streaming, 16 bits
        _run("cavity_d3q27_kbc_256", "D3Q27", (256, 256, 256), "8,8,4", 50, "cavity", tau=0.50765, f16=True,
             arith="fast", method="eso", coll="KBC", les="smagorinsky"),
        # large-eddy simulation of a decaying vortex on an ordinary grid
        _run("tgv_smagorinsky_128", "D3Q19", (128, 128, 128), "8,8,4", 200, "tgv", tau=0.501910, les="smagorinsky",
             U=0.05),
        # the same flow with the trained closure, at the size it was trained for
        _run("tgv_learned_256", "D3Q19", (256, 256, 256), "8,8,4", 50, "tgv", tau=0.503820, les="learned", U=0.05),
        # a grid whose sides no tile divides: the untiled layout, LBM_Grid's default
        _run("cavity_d3q19_untiled", "D3Q19", (150, 131, 97), "untiled", 50, "cavity", tau=0.8),
        # parameter study: many uneven cylinder channels in one batch
        dict(name="batch_channels_128", kind="batch", domains=128, specs=0, tile="32,8,1", steps=64),
        # training of the closure: one mini-batch of the shipped training loop
        dict(name="train_closure", kind="train", rows=1 << 18),
        # what a program writes out between runs
        dict(name="outputs_256", kind="outputs", lattice="D3Q19", nx=256, ny=256, nz=256, tile="8,8,4", method="db",
             f16=False, tau=0.8, U=0.1, flow="cavity"),
        # what every run begins with
        dict(name="setup_256", kind="setup", lattice="D3Q19", nx=256, ny=256, nz=256, tile="8,8,4", method="db",
             f16=False, tau=0.8, U=0.1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng, lattice, lo, hi):
    """(shape, tile): the default tiles' multiples, other 256-cell tiles, and odd untiled shapes."""
    two_d = lattice == "D2Q9"
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = cells ** (0.5 if two_d else 1.0 / 3.0)
    tile = rng.choice(["16,16,1", "32,8,1", "untiled"] if two_d else ["8,8,4", "8,8,4", "16,4,4", "untiled"])
    t = (1, 1, 1) if tile == "untiled" else tuple(int(v) for v in tile.split(","))
    stretch = [math.exp(rng.uniform(-0.4, 0.4)) for _ in range(3)]
    shape = [max(2, int(round(side * stretch[d] / t[d]))) * t[d] for d in range(3)]
    if two_d:
        shape[2] = 1
    return tuple(shape), tile


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["loop", "batch", "train", "outputs", "setup"])
    if kind == "run":
        lattice = rng.choice(["D2Q9", "D3Q19", "D3Q19", "D3Q27"])
        shape, tile = _draw_grid(rng, lattice, 2e4, 1.2e7)
        cells = shape[0] * shape[1] * shape[2]
        coll = rng.choice(["SRT", "SRT", "TRT", "RLBM", "KBC"])
        f16 = rng.random() < 0.4
        les = rng.choice(["off", "off", "smagorinsky"])
        if lattice == "D3Q19" and tile != "untiled" and rng.random() < 0.2:
            les, coll, f16 = "learned", "SRT", False
        flow = "tgv" if les == "learned" else rng.choice(["cavity", "cavity", "periodic"])
        if flow == "tgv":  # a cube of whole tiles
            n = max(32, 16 * int(round(cells ** (1.0 / 3.0) / 16)))
            shape, cells = (n, n, n), n ** 3
        steps = 2 * max(10, min(400, int(LARGEST / cells / 4)))
        arith = "exact" if les == "learned" else rng.choice(["exact", "fast"])
        method = "db" if les == "learned" else rng.choice(["db", "db", "eso"])
        # the trained closure belongs to one relaxation time and amplitude
        tau, U = (0.50382, 0.05) if les == "learned" else (round(rng.uniform(0.55, 1.3), 4), round(rng.uniform(0.02, 0.1), 4))
        return _run(None, lattice, shape, tile, min(steps, _log_int(rng, 20, 800) // 2 * 2), flow, coll=coll, f16=f16,
                    les=les, arith=arith, method=method, tau=tau, U=U)
    if kind == "loop":
        ny = 16 * _log_int(rng, 4, 24)
        return dict(kind="loop", nx=16 * int(round(ny * 2.5 / 16)), ny=ny, steps=2 * rng.randint(4, 16),
                    Re=round(rng.uniform(20.0, 100.0), 2), offset=round(rng.uniform(-0.05, 0.05), 4))
    if kind == "batch":
        return dict(kind="batch", domains=_log_int(rng, 4, 128), specs=rng.randrange(1 << 20),
                    tile=rng.choice(["32,8,1", "16,16,1"]), steps=2 * rng.randint(8, 48))
    if kind == "train":
        return dict(kind="train", rows=_log_int(rng, 1 << 12, 1 << 20))
    lattice = rng.choice(["D2Q9", "D3Q19", "D3Q27"])
    shape, tile = _draw_grid(rng, lattice, 1e5, 1e7)
    case = dict(kind=kind, lattice=lattice, nx=shape[0], ny=shape[1], nz=shape[2], tile=tile,
                method=rng.choice(["db", "eso"]), f16=rng.random() < 0.3, tau=round(rng.uniform(0.55, 1.3), 4),
                U=round(rng.uniform(0.02, 0.1), 4))
    if kind == "outputs":
        case["flow"] = rng.choice(["cavity", "periodic"])
    return case


# ---- set-up ------------------------------------------------------------------------------------


def _grid(case):
    tile = case["tile"] if case["tile"] == "untiled" else tuple(int(v) for v in case["tile"].split(","))
    return LBM_Grid(get_lattice(LATTICE[case["lattice"]]), case["nx"], case["ny"], case["nz"], tile)


def _config(case):
    method = LBM_method.DOUBLE_BUFFER if case["method"] == "db" else LBM_method.ESOTERIC_PULL
    return LBM_Config(method, collision_op=case.get("coll", "SRT"), LES=case.get("les", "off") != "off",
                      DDF_shift=case["f16"], use_float16c=case["f16"],
                      include_moving_boundary=case.get("flow", "cavity") == "cavity", arithmetic=case.get("arith", "exact"))


def _velocity(shape, D, amp, seed):
    """A smooth random velocity field [D, nx, ny, nz] (three low-wavenumber waves per component)."""
    rng = np.random.default_rng(seed)
    ax = [torch.arange(n, device=DEV, dtype=torch.float64) * (2 * math.pi / n) for n in shape]
    u = torch.zeros((D,) + tuple(shape), dtype=torch.float64, device=DEV)
    for d in range(D):
        for _ in range(3):
            k, ph = rng.integers(1, 3, size=3), rng.uniform(0, 2 * math.pi)
            arg = (k[0] * ax[0])[:, None, None] + (k[1] * ax[1])[None, :, None] + ((k[2] * ax[2])[None, None, :] + ph)
            u[d] += amp / 3 * torch.sin(arg)
    return u.float().contiguous()


def _initial(case, seed):
    """(u, grad or None) of the initial state."""
    grid_D = 2 if case["lattice"] == "D2Q9" else 3
    if case.get("flow") == "tgv":
        return tgv.tgv_fields(case["nx"], case["U"], seed=seed, device=DEV)
    return _velocity((case["nx"], case["ny"], case["nz"]), grid_D, 0.5 * case["U"], seed), None


SIDES = ("-Y", "+X", "-X", "+Z", "-Z", "+Y")  # the lid last


def _paint(grid, cfg, flags, bc, U):
    for side in SIDES:
        if grid.D == 3 or side[1] != "Z":
            u = [U if side == "+Y" else 0.0] + [0.0] * (grid.D - 1)
            preprocess.set_exterior_walls(grid, cfg, flags, bc, side, Flags.SOLID, u, 1.0)


def _domain(case, seed):
    grid, cfg = _grid(case), _config(case)
    n = grid.num_points
    s = dict(case=case, grid=grid, cfg=cfg, solver=Solver(grid, cfg))
    s["flags"] = torch.zeros(n, dtype=torch.uint8, device=DEV)
    s["bc"] = torch.zeros(n * (grid.D + 1), device=DEV)
    if case["flow"] == "cavity":
        _paint(grid, cfg, s["flags"], s["bc"], case["U"])
    s["f"] = torch.zeros(n * grid.Q, dtype=torch.int16 if case["f16"] else torch.float32, device=DEV)
    u, grad = _initial(case, seed)
    s["solver"].init_equilibrium(s["f"], 1.0, case["tau"], u, grad)
    s["f2"] = s["f"].clone() if case["method"] == "db" else None
    s["rho"] = torch.zeros(grid.shape, device=DEV)
    s["u"] = torch.zeros((grid.D,) + grid.shape, device=DEV)
    if case["f16"]:
        s["populations"] = torch.empty(n * grid.Q, device=DEV)
    return s


def _channels(case):
    if case["kind"] == "loop":
        return [workloads.Channel(case["nx"], case["ny"], case["Re"], 0.05, case["offset"], (16, 16, 1))]
    specs = workloads.channel_specs(case["domains"], seed=case["specs"], granule=(32, 32))
    return workloads.cylinder_channels(tile=tuple(int(v) for v in case["tile"].split(",")), specs=specs)


def _net_rows(case, seed):
    """(rows, targets, output scale): normalised features and positive targets, as the training loop has them."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn((case["rows"], closure.N_FEATURES), device=DEV, generator=g).clamp_(-4, 4)
    w = torch.randn(closure.N_FEATURES, device=DEV, generator=g)
    nu = 1e-4 * torch.exp(0.3 * (x * w).sum(1))
    return x, nu.contiguous(), 1e-4


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "outputs"):
        s = _domain(case, seed)
        if case.get("les") == "learned":
            closure.set_closure(s["solver"], closure.LearnedClosure.load(CLOSURE_FILE, device=DEV))
        if kind == "outputs":
            s["q"] = torch.zeros(s["grid"].shape, device=DEV)
        return s
    if kind == "loop":
        ch = _channels(case)[0]
        solver, asm = Solver(ch.grid, ch.cfg), Assembly(ch.grid, ch.cfg)
        asm.flags_host[:], asm.bc_host[:] = ch.flags, ch.bc
        asm.upload()
        u = _velocity(ch.grid.shape, 2, 0.02, seed)
        solver.init_equilibrium(asm.f, 1.0, ch.tau, u)
        asm.f2.copy_(asm.f)
        b = ch.body
        body = geometry.RigidStationaryObject(ch.grid, b.unique_fluid_ids, b.fluid_boundaries_list,
                                              b.lattice_links_list, b.link_distances_list)
        return dict(case=case, solver=solver, asm=asm, body=body, tau=ch.tau)
    if kind == "batch":
        chans = _channels(case)
        batch = BatchSolver([c.grid for c in chans], chans[0].cfg)
        off = np.concatenate([[0], np.cumsum([c.grid.num_points for c in chans])]).astype(np.int64)
        f = torch.empty(int(off[-1]) * 9, device=DEV)
        bc = torch.from_numpy(np.concatenate([c.bc for c in chans])).to(DEV)
        flags = torch.from_numpy(np.concatenate([c.flags for c in chans])).to(DEV)
        for i, c in enumerate(chans):
            fi = f[9 * off[i]:9 * off[i + 1]]
            Solver(c.grid, c.cfg).init_equilibrium(fi, 1.0, c.tau, _velocity(c.grid.shape, 2, 0.02, seed + i))
        f2 = f.clone()
        for i, c in enumerate(chans):
            a, b = int(off[i]), int(off[i + 1])
            batch.set_domain(i, f[9 * a:9 * b], f2[9 * a:9 * b], bc[3 * a:3 * b], flags[a:b], c.tau)
        dom, ids, dirs, dists, method = workloads.links_of(chans, DEV)
        force = torch.zeros(ids.numel() * 2, device=DEV)
        batch.set_links(dom, ids, dirs, dists, method, 0.0, force)
        return dict(case=case, batch=batch, f=f, f2=f2, bc=bc, flags=flags, force=force)
    if kind == "train":
        x, nu, scale = _net_rows(case, seed)
        theta = closure.init_theta(seed % 1000, device=DEV)
        return dict(case=case, x=x, target=nu, scale=scale, theta=theta, opt=closure.Adam(theta, lr=3e-3))
    if kind == "setup":
        grid, cfg = _grid(case), _config(case)
        n, D = grid.num_points, grid.D
        u = _velocity(grid.shape, D, 0.5 * case["U"], seed)
        return dict(case=case, grid=grid, cfg=cfg, solver=Solver(grid, cfg), u=u,
                    grad=_velocity(grid.shape, D * D, 1e-3, seed + 1),
                    flags=torch.zeros(n, dtype=torch.uint8, device=DEV), bc=torch.zeros(n * (D + 1), device=DEV),
                    f=torch.zeros(n * grid.Q, dtype=torch.int16 if case["f16"] else torch.float32, device=DEV),
                    populations=torch.empty(n * grid.Q, device=DEV) if case["f16"] else None)
    raise ValueError(kind)


# ---- one pass ----------------------------------------------------------------------------------


def _populations(s):
    """The state's populations as float32: the lattice itself, or its Float16C codes decoded."""
    if not s["case"]["f16"]:
        return s["f"]
    _capi.check(_capi.lib().lbm_float16c_decode(_capi.ptr(s["f"]), _capi.ptr(s["populations"]), s["f"].numel(), None))
    return s["populations"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        solver = s["solver"]
        solver.run(s["f"], s["f2"], s["bc"], s["flags"], case["tau"], case["steps"], 0)
        solver.compute_rho_u(s["rho"], s["u"], s["f"], s["bc"], s["flags"], after_odd_step=True)
        return {"f": _populations(s), "rho": s["rho"], "u": s["u"]}
    if kind == "loop":
        solver, asm, body = s["solver"], s["asm"], s["body"]
        for k in range(0, case["steps"], 2):
            solver.even_step(asm, s["tau"])
            body.bounceback(solver, asm.f2, 1, True)
            solver.odd_step(asm, s["tau"])
            body.bounceback(solver, asm.f, 1, True)
        return {"f": asm.f, "forces": body.link_forces, "force": list(body.sum_force(solver))}
    if kind == "batch":
        s["batch"].run(case["steps"], 0)
        return {"f": s["f"], "force": s["force"]}
    if kind == "train":
        th = s["theta"].detach().requires_grad_(True)
        nu = closure.mlp(th, s["x"], s["scale"])
        loss = (((nu - s["target"]) / s["scale"]) ** 2).mean()
        loss.backward()
        s["opt"].step(th.grad)
        return {"nu": nu.detach(), "grad": th.grad, "theta": s["theta"]}
    if kind == "outputs":
        solver = s["solver"]
        solver.compute_rho_u(s["rho"], s["u"], s["f"], s["bc"], s["flags"], after_odd_step=True)
        solver.q_criterion(s["q"], s["f"], s["bc"], s["flags"], s["u"], case["tau"], after_odd_step=True)
        total = solver.mass_momentum(s["f"], s["flags"], after_odd_step=True)
        return {"rho": s["rho"], "u": s["u"], "q": s["q"], "mass": total[0]}
    if kind == "setup":
        _paint(s["grid"], s["cfg"], s["flags"], s["bc"], case["U"])
        _body(s)
        s["solver"].init_equilibrium(s["f"], 1.0, case["tau"], s["u"], s["grad"])
        return {"flags": s["flags"], "bc": s["bc"], "f": _populations(s)}
    raise ValueError(kind)


def _body(s):
    """A sphere (a circle in 2D) and a box in the painted domain."""
    nx, ny, nz = s["grid"].shape
    add = geometry.add_sphere if s["grid"].D == 3 else geometry.add_circle
    add(s["grid"], s["flags"], [0.3 * nx, 0.5 * ny, 0.5 * nz if nz > 1 else 0.0], 0.1 * ny)
    geometry.add_box(s["grid"], s["flags"], [0.7 * nx, 0.5 * ny, 0.5 * nz if nz > 1 else 0.0],
                     [0.05 * nx, 0.1 * ny, 0.1 * nz if nz > 1 else 0.0])


# ---- what a pass cannot do without -------------------------------------------------------------


def _flops_per_update(Q, coll, les):
    """Float operations of one cell update in the shortest form of the operator: moments, equilibria and relaxation per
    direction, plus the stress of LES, RLBM and KBC."""
    n = 9 * Q + 20
    if les != "off" or coll in ("RLBM", "KBC"):
        n += 4 * Q + 20
    if coll == "KBC":
        n += 8 * Q
    return n + (2624 if les == "learned" else 0)


def work(case):
    kind = case["kind"]
    if kind in ("run", "outputs", "setup"):
        Q, D = (9, 2) if case["lattice"] == "D2Q9" else (19 if case["lattice"] == "D3Q19" else 27, 3)
        n = case["nx"] * case["ny"] * case["nz"]
        lattice = n * Q * (2 if case["f16"] else 4)
        decoded = n * Q * 4 if case["f16"] else 0
        if kind == "run":
            flops = n * case["steps"] * _flops_per_update(Q, case["coll"], case["les"])
            return {"bytes": 2 * lattice + n + 4 * n * (D + 1) + decoded, "flops": flops}
        if kind == "outputs":
            return {"bytes": lattice + n + 4 * n * (D + 2), "flops": n * (15 * Q + 60)}
        return {"bytes": lattice + n + 4 * n * (D + D * D) + decoded, "flops": n * 12 * Q}
    if kind == "loop":
        n = case["nx"] * case["ny"]
        return {"bytes": n * (72 + 13), "flops": n * case["steps"] * _flops_per_update(9, "SRT", "off")}
    if kind == "batch":
        specs = workloads.channel_specs(case["domains"], seed=case["specs"], granule=(32, 32))
        n = sum(nx * ny for nx, ny, _, _ in specs)
        return {"bytes": n * (72 + 13), "flops": n * case["steps"] * _flops_per_update(9, "SRT", "off")}
    return {"bytes": case["rows"] * 4 * 10, "flops": case["rows"] * 6 * 1312}


# ---- the same pass in 64 bits ------------------------------------------------------------------


class _Lattice64:
    """Directions and weights of a lattice (rest, then opposite pairs), from their definition."""

    def __init__(self, name):
        if name == "D2Q9":
            c = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (-1, 1, 0)]
            w = {0: 4 / 9, 1: 1 / 9, 2: 1 / 36}
        else:
            c = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1),
                 (0, 1, -1)]
            w = {0: 1 / 3, 1: 1 / 18, 2: 1 / 36}
            if name == "D3Q27":
                c += [(1, 1, 1), (1, 1, -1), (1, -1, 1), (-1, 1, 1)]
                w = {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}
        full = [c[0]]
        for v in c[1:]:
            full += [v, tuple(-a for a in v)]
        self.c, self.Q, self.D = full, len(full), 2 if name == "D2Q9" else 3
        self.w = [w[sum(abs(a) for a in v)] for v in full]
        self.opp = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, self.Q)]
        self.pairs = [(a, b) for a in range(self.D) for b in range(a, self.D)]

    def cu(self, q, u):
        return sum(self.c[q][d] * u[d] for d in range(self.D) if self.c[q][d]) if q else torch.zeros_like(u[0])

    def feq(self, q, rho, u, uu, shift):
        cu = self.cu(q, u)
        e = self.w[q] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu)
        return e - self.w[q] if shift else e


def _natural(flat, K, shape, tile):
    """[K, nx, ny, nz] of a flat tiled array."""
    t = shape if tile == "untiled" else tuple(int(v) for v in tile.split(","))
    n = [a // b for a, b in zip(shape, t)]
    a = flat.reshape(n[2], n[1], n[0], K, t[2], t[1], t[0]).permute(3, 2, 6, 1, 5, 0, 4)
    return a.reshape((K,) + tuple(shape))


def _tiled(a, tile):
    """The flat tiled array of a [K, nx, ny, nz] one."""
    K, shape = a.shape[0], tuple(a.shape[1:])
    t = shape if tile == "untiled" else tuple(int(v) for v in tile.split(","))
    n = [p // q for p, q in zip(shape, t)]
    v = a.reshape(K, n[0], t[0], n[1], t[1], n[2], t[2]).permute(5, 3, 1, 0, 6, 4, 2)
    return v.reshape(-1)


class _Flow64:
    """One domain in float64: flags and boundary values as given, populations [Q, nx, ny, nz]."""

    def __init__(self, lattice, flags, bc, tau, *, shift=False, moving=True, method="db", coll="SRT", les="off"):
        self.L, self.tau = _Lattice64(lattice), float(np.float32(tau))
        self.flags, self.bc = flags, bc.double()
        self.shift, self.moving, self.method, self.coll, self.les = shift, moving, method, coll, les
        self.solid = flags == Flags.SOLID
        self.eq = flags == Flags.EQUILIBRIUM
        self.any_solid, self.any_eq = bool(self.solid.any()), bool(self.eq.any())
        self.net = None

    def at(self, a, c, sign=1):
        """a at x + sign * c (periodic)."""
        s = [-sign * v for v in c]
        return torch.roll(a, s, (-3, -2, -1)) if any(s) else a

    def init(self, u, grad):
        L, rho = self.L, torch.ones_like(u[0], dtype=torch.float64)
        u = u.double()
        uu = (u * u).sum(0)
        f = torch.stack([L.feq(q, rho, u, uu, self.shift) for q in range(L.Q)])
        if grad is not None:
            g, tau = grad.double(), self.tau
            for q in range(L.Q):
                n = torch.zeros_like(uu)
                for a in range(L.D):
                    for b in range(L.D):
                        k = L.c[q][a] * L.c[q][b] - (1 / 3 if a == b else 0.0)
                        n += k * 0.5 * (g[a * L.D + b] + g[b * L.D + a])
                f[q] += n * (-L.w[q] * tau * 3.0) * ((tau - 1.0) / tau)
        return self.scatter(f, odd=True) if self.method == "eso" else f

    def scatter(self, f, odd, into=None):
        """The in-place method's store: f[pos] to x + c in slot pos (odd) or neg, f[neg] to x in the other."""
        out = torch.zeros_like(f) if into is None else into
        live = ~self.solid
        put = (lambda old, new, m: new) if into is None or not self.any_solid else (lambda o, n, m: torch.where(m, n, o))
        out[0] = put(out[0], f[0], live)
        for p in range(1, self.L.Q, 2):
            c = self.L.c[p]
            far, near = (p, p + 1) if odd else (p + 1, p)
            out[far] = put(out[far], self.at(f[p], c, -1), self.at(live, c, -1))
            out[near] = put(out[near], f[p + 1], live)
        return out

    def gather(self, f, even):
        """Populations a cell loads in the next step (in-place method)."""
        g = torch.empty_like(f)
        g[0] = f[0]
        for p in range(1, self.L.Q, 2):
            a, b = (p, p + 1) if even else (p + 1, p)
            g[p], g[p + 1] = f[a], self.at(f[b], self.L.c[p])
        return g

    def pulled(self, f, even):
        """Streamed populations with the boundary conditions applied."""
        L = self.L
        if self.method == "eso":
            g = self.gather(f, even)
        else:
            g = torch.stack([self.at(f[q], L.c[q], -1) for q in range(L.Q)])
        if self.any_solid:
            for q in range(1, L.Q):
                wall = self.at(self.solid, L.c[q], -1)
                if self.method == "db":
                    g[q] = torch.where(wall, f[L.opp[q]], g[q])
                if self.moving:
                    push = 6 * L.w[q] * self.bc[L.D] * sum(L.c[q][d] * self.bc[d] for d in range(L.D) if L.c[q][d])
                    g[q] = torch.where(wall, g[q] + self.at(push, L.c[q], -1), g[q])
        if self.any_eq:
            h = g.clone()
            for q in range(1, L.Q):
                for d in range(L.D):
                    if L.c[q][d]:
                        edge = [slice(None)] * 3
                        edge[d] = 0 if L.c[q][d] > 0 else -1
                        h[(q,) + tuple(edge)] = 0.0 if self.shift else L.w[q]
            rho, u = self.moments(h)
            free = torch.isnan(self.bc[0])
            u = torch.where(free, u, self.bc[: L.D])
            rho = torch.where(torch.isnan(self.bc[L.D]), rho, self.bc[L.D])
            uu = (u * u).sum(0)
            for q in range(L.Q):
                g[q] = torch.where(self.eq, L.feq(q, rho, u, uu, self.shift), g[q])
        return g

    def moments(self, f):
        rho = f.sum(0) + (1.0 if self.shift else 0.0)
        m = torch.zeros((self.L.D,) + tuple(rho.shape), dtype=f.dtype, device=f.device)
        for q in range(1, self.L.Q):
            for d in range(self.L.D):
                if self.L.c[q][d]:
                    m[d] += self.L.c[q][d] * f[q]
        return rho, m / rho

    def stress(self, f, rho, u, uu):
        L = self.L
        P = [torch.zeros_like(rho) for _ in L.pairs]
        for q in range(L.Q):
            n = f[q] - L.feq(q, rho, u, uu, self.shift)
            for k, (a, b) in enumerate(L.pairs):
                if L.c[q][a] * L.c[q][b]:
                    P[k] = P[k] + L.c[q][a] * L.c[q][b] * n
        return P

    def strain(self, P, rho):
        S = [-p / (2 * rho / 3 * self.tau) for p in P]
        s2 = sum(s * s * (1 if a == b else 2) for s, (a, b) in zip(S, self.L.pairs))
        return S, s2

    def collide(self, f):
        L = self.L
        rho, u = self.moments(f)
        uu = (u * u).sum(0)
        tau = torch.full_like(rho, self.tau)
        if self.les != "off" or self.coll in ("RLBM", "KBC"):
            P = self.stress(f, rho, u, uu)
        if self.les != "off":
            S, s2 = self.strain(P, rho)
            smag = float(np.float32(0.1)) ** 2 * torch.sqrt(2 * s2)
            tau = tau + 3 * (smag if self.les == "smagorinsky" else self.learned(S, s2, rho, uu, smag))
        eq = [L.feq(q, rho, u, uu, self.shift) for q in range(L.Q)]
        out = torch.empty_like(f)
        if self.coll == "SRT":
            for q in range(L.Q):
                out[q] = f[q] - (f[q] - eq[q]) / tau
        elif self.coll == "TRT":
            ta = 0.5 + 0.1875 / (tau - 0.5)
            out[0] = f[0] - (f[0] - eq[0]) / tau
            for q in range(1, L.Q, 2):
                s = ((f[q] + f[q + 1]) - (eq[q] + eq[q + 1])) / (2 * tau)
                a = ((f[q] - f[q + 1]) - (eq[q] - eq[q + 1])) / (2 * ta)
                out[q], out[q + 1] = f[q] - s - a, f[q + 1] - s + a
        elif self.coll == "RLBM":
            for q in range(L.Q):
                dot = sum(P[k] * (2 * L.c[q][a] * L.c[q][b] if a != b else L.c[q][a] ** 2 - 1 / 3)
                          for k, (a, b) in enumerate(L.pairs))
                out[q] = eq[q] + (1 - 1 / tau) * 4.5 * L.w[q] * dot
        else:
            beta, sp, hp = 1 / (2 * tau), torch.zeros_like(rho), torch.zeros_like(rho)
            ds = [self.shear(q, P) for q in range(L.Q)]
            for q in range(L.Q):
                dh = f[q] - eq[q] - ds[q]
                e = eq[q] + L.w[q] if self.shift else eq[q]
                sp, hp = sp + ds[q] * dh / e, hp + dh * dh / e
            gamma = 1 / beta - (2 - 1 / beta) * sp / (hp + 1e-32)
            for q in range(L.Q):
                out[q] = f[q] - beta * (2 * ds[q] + gamma * (f[q] - eq[q] - ds[q]))
        return out

    def shear(self, q, P):
        """Shear part of a population: the deviatoric stress on the lattice's second-order polynomials."""
        c, n = self.L.c[q], sum(abs(a) for a in self.L.c[q])
        if n == 2:
            a, b = [d for d in range(3) if c[d]]
            return c[a] * c[b] * P[self.L.pairs.index((a, b))] / 4
        if n != 1:
            return torch.zeros_like(P[0])
        if self.L.D == 2:
            return (P[0] - P[2]) * (0.25 if c[0] else -0.25)
        d = next(d for d in range(3) if c[d])
        return ((3 * P[(0, 3, 5)[d]]) - (P[0] + P[3] + P[5])) / 6

    def learned(self, S, s2, rho, uu, smag):
        """Eddy viscosity of the trained network, the Smagorinsky one outside its training range."""
        n, q = self.net, 2 * s2 + 1e-24
        r, tr = 1 / torch.sqrt(q), S[0] + S[3] + S[5]
        a, b, c = S[0] - tr / 3, S[3] - tr / 3, S[5] - tr / 3
        det = a * (b * c - S[4] ** 2) - S[1] * (S[1] * c - S[4] * S[2]) + S[2] * (S[1] * S[4] - b * S[2])
        off = S[1] ** 2 + S[2] ** 2 + S[4] ** 2
        x = torch.stack([torch.log(q) / 2, tr * r, det * r ** 3, rho - 1, torch.sqrt(uu), 4 * off * r * r,
                         torch.full_like(q, math.log(self.tau - 0.5)), uu * r], -1)
        x = ((x - n["mean"]) * n["scale"]).reshape(-1, 8)
        inside = ((x >= n["lo"]) & (x <= n["hi"])).all(1)
        nu = torch.cat([_net64(n["theta"], part)[0] for part in x.split(1 << 21)]) * n["nu_scale"]
        return torch.where(inside, nu, smag.reshape(-1)).reshape(q.shape)

    def step(self, f, even=True):
        g = self.collide(self.pulled(f, even))
        if self.method == "eso":
            return self.scatter(g, odd=not even, into=f)
        return torch.where(self.solid, f, g) if self.any_solid else g

    def fields(self, f):
        g = self.pulled(f, True)
        rho, u = self.moments(g)
        if self.any_solid:
            rho = torch.where(self.solid, self.bc[self.L.D], rho)
            u = torch.where(self.solid, self.bc[: self.L.D], u)
        return g, rho, u

    def difference(self, a, d):
        """The velocity gradient of the Q-criterion: one-sided differences over 1 cell, 1/2 towards a solid one, each
        weighted by the other's share; 0 at an edge of the grid."""
        def side(sign):
            c = [sign if k == d else 0 for k in range(3)]
            h = torch.where(self.at(self.solid, c), 0.5, 1.0).double()
            g = sign * (self.at(a, c) - a) / h
            edge = [slice(None)] * 3
            edge[d] = -1 if sign > 0 else 0
            h[tuple(edge)], g[tuple(edge)] = 0.0, 0.0
            return g, h
        (gl, hl), (gr, hr) = side(-1), side(1)
        lw = 1 - hl / (hl + hr)
        return gr * (1 - lw) + gl * lw

    def q_criterion(self, g, u):
        rho, v = self.moments(g)
        _, s2 = self.strain(self.stress(g, rho, v, (v * v).sum(0)), rho)
        w2 = (self.difference(u[1], 0) - self.difference(u[0], 1)) ** 2
        if self.L.D == 3:
            w2 = w2 + (self.difference(u[2], 1) - self.difference(u[1], 2)) ** 2
            w2 = w2 + (self.difference(u[0], 2) - self.difference(u[2], 0)) ** 2
        return torch.where(self.solid, 0.0, 0.25 * w2 - 0.5 * s2)


def _net64(theta, x):
    """(softplus output, pre-activations) of the 8-32-32-1 network in float64."""
    w1, b1, w2, b2, w3, b3 = torch.split(theta, [256, 32, 1024, 32, 32, 1])
    h = torch.relu(x @ w1.reshape(8, 32) + b1)
    h = torch.relu(h @ w2.reshape(32, 32) + b2)
    y = h @ w3 + b3
    return torch.nn.functional.softplus(y, threshold=1e9), y


def _walls64(case, body=False):
    """(flags, bc) [nx, ny, nz] and [D + 1, nx, ny, nz] of a cavity (or an open periodic box)."""
    shape, D = (case["nx"], case["ny"], case["nz"]), 2 if case["lattice"] == "D2Q9" else 3
    flags = torch.zeros(shape, dtype=torch.uint8, device=DEV)
    bc = torch.zeros((D + 1,) + shape, dtype=torch.float32, device=DEV)
    if case.get("flow", "cavity") == "cavity":
        for side in SIDES:
            if D == 3 or side[1] != "Z":
                at = [slice(None)] * 3
                at["XYZ".index(side[1])] = 0 if side[0] == "-" else -1
                flags[tuple(at)] = Flags.SOLID
                bc[(slice(None),) + tuple(at)] = 0.0
                bc[(D,) + tuple(at)] = 1.0
                if side == "+Y":
                    bc[(0,) + tuple(at)] = case["U"]
    return flags, bc


def _flow64(case):
    flags, bc = _walls64(case)
    return _Flow64(case["lattice"], flags, bc, case["tau"], shift=case["f16"], moving=case.get("flow", "cavity") == "cavity",
                   method=case["method"], coll=case.get("coll", "SRT"), les=case.get("les", "off"))


def _links64(f, lat, dom, forces, at0):
    """Link-wise interpolated bounce-back in place on f [Q, nx, ny, nz]; the link forces into forces[:, at0:]."""
    n = len(dom["ids"])
    if n == 0:
        return
    x, y, i, q = dom["x"], dom["y"], dom["dirs"], dom["dists"]
    c = torch.tensor([v[:2] for v in lat.c], device=DEV)
    opp = torch.tensor(lat.opp, device=DEV)[i]
    into = f[i, x, y, 0]
    far = f[opp, (x - c[i, 0]) % f.shape[1], (y - c[i, 1]) % f.shape[2], 0]
    bb = torch.where(q > 0.5, 0.5 / q * into + (2 * q - 1) / (2 * q) * f[opp, x, y, 0], 2 * q * into + (1 - 2 * q) * far)
    f[i, x, y, 0] = bb
    forces[:, at0:at0 + n] = c[i].T * (into + bb)


def _channels64(case, seed):
    """(f, forces [2, links]) of the channels after the pass."""
    chans, out, at0 = _channels(case), [], 0
    forces = torch.zeros((2, sum(c.body.num_links() for c in chans)), dtype=torch.float64, device=DEV)
    for k, ch in enumerate(chans):
        tile = "%d,%d,%d" % ch.grid.tile_shape
        shape = ch.grid.shape
        flags = _natural(torch.from_numpy(ch.flags).to(DEV), 1, shape, tile)[0]
        bc = _natural(torch.from_numpy(ch.bc).to(DEV), 3, shape, tile)
        flow = _Flow64("D2Q9", flags, bc, ch.tau)
        xy = torch.stack(torch.meshgrid(*[torch.arange(n, device=DEV) for n in shape], indexing="ij"))
        xy = torch.stack([_tiled(xy[d][None], tile) for d in range(2)])
        ids = torch.from_numpy(ch.body.fluid_boundaries_list.astype(np.int64)).to(DEV)
        dom = dict(ids=ids, x=xy[0][ids], y=xy[1][ids],
                   dirs=torch.from_numpy(ch.body.lattice_links_list.astype(np.int64)).to(DEV),
                   dists=torch.from_numpy(ch.body.link_distances_list).to(DEV).double())
        f = flow.init(_velocity(shape, 2, 0.02, seed + k), None)
        for _ in range(case["steps"]):
            f = flow.step(f)
            _links64(f, flow.L, dom, forces, at0)
        out.append(_tiled(f, tile))
        at0 += len(ids)
    return torch.cat(out), forces


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        flow = _flow64(case)
        if case["les"] == "learned":
            d = np.load(CLOSURE_FILE)
            flow.net = {k: torch.tensor(d[k], dtype=torch.float64, device=DEV) for k in ("theta", "mean", "scale", "lo", "hi")}
            flow.net["nu_scale"] = float(d["nu_scale"])
        f = flow.init(*_initial(case, seed))
        for k in range(case["steps"]):
            f = flow.step(f, even=k % 2 == 0)
        _, rho, u = flow.fields(f)
        return {"f": _tiled(f, case["tile"]), "rho": rho, "u": u}
    if kind == "loop":
        f, forces = _channels64(case, seed)
        return {"f": f, "forces": forces.reshape(-1), "force": [float(v) for v in forces.sum(1)]}
    if kind == "batch":
        f, forces = _channels64(case, seed)
        return {"f": f, "force": forces.reshape(-1)}
    if kind == "train":
        x, target, scale = _net_rows(case, seed)
        theta = closure.init_theta(seed % 1000, device=DEV).double().requires_grad_(True)
        nu = _net64(theta, x.double())[0] * scale
        ((((nu - target.double()) / scale) ** 2).mean()).backward()
        g = theta.grad
        # the first step of Adam from zero moments: lr g / (|g| + eps)
        new = theta.detach() - 3e-3 * g / (g.abs() + 1e-8)
        return {"nu": nu.detach(), "grad": g, "theta": new}
    if kind == "outputs":
        flow = _flow64(case)
        f = flow.init(*_initial(case, seed))
        g, rho, u = flow.fields(f)
        q = flow.q_criterion(g, u)
        live = ~flow.solid
        if case["method"] == "eso":  # the populations a cell owns after an odd step
            own = torch.empty_like(f)
            own[0] = f[0]
            for p in range(1, flow.L.Q, 2):
                own[p], own[p + 1] = flow.at(f[p], flow.L.c[p]), f[p + 1]
            f = own
        mass = float((f.sum(0) + (1.0 if flow.shift else 0.0))[live].sum())
        return {"rho": rho, "u": u, "q": q, "mass": mass}
    if kind == "setup":
        flow = _flow64(case)
        flow.solid = torch.zeros_like(flow.solid)  # the initial state fills every cell
        f = flow.init(_velocity(tuple(flow.flags.shape), flow.L.D, 0.5 * case["U"], seed),
                      _velocity(tuple(flow.flags.shape), flow.L.D ** 2, 1e-3, seed + 1))
        return {"flags": None, "bc": _tiled(flow.bc, case["tile"]), "f": _tiled(f, case["tile"])}
    return None
