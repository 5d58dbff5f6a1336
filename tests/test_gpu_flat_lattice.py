"""D2Q9 on grids that extend along z and x or y only (accepted: the number of extents above 1 is what is
checked).  The reference's 2D neighbours are those of the plane z = 0 (get_adjacent_idx), which the oracle
restates: the generic step in calls that gather the flags and in runs that use masks, the initial state and
the outputs give the oracle's words in every plane."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu

GRIDS = [((32, 1, 32), "untiled"), ((33, 1, 9), (3, 1, 9)), ((24, 1, 40), (4, 1, 5)), ((1, 16, 12), "untiled"),
         ((1, 50, 6), (1, 5, 2))]


def _case(shape, tile, meth, f16, kind):
    grid = make_grid("D2Q9", shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points)
    flags, bc = mixed_flags(grid, rng)
    if kind == "fluid":
        flags[:] = 0
    return grid, cfg, rng, flags, bc


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("kind", ["fluid", "mixed"])
@pytest.mark.parametrize("shape,tile", GRIDS)
def test_steps(shape, tile, kind, f16):
    grid, cfg, rng, flags, bc = _case(shape, tile, "db", f16, kind)
    f = initial_f(grid, cfg, rng)
    f2 = f.copy()
    a, b, fl, bcd = to_dev(f), to_dev(f), to_dev(flags), to_dev(bc)
    s = Solver(grid, cfg)
    s.set_kernel_path(1)
    for n in (2, 32):
        s.run(a, b, bcd, fl, 0.8, n, 0)
        for _ in range(n):
            oracle.step(cfg, grid, 32, f2, f, bc, flags, 0.8)
            f, f2 = f2, f
        word = np.uint16 if f16 else np.uint32
        assert np.array_equal(a.cpu().numpy().view(word), f.view(word)), n


@pytest.mark.parametrize("meth,f16", [("db", False), ("eso", True)])
@pytest.mark.parametrize("kind", ["fluid", "mixed"])
@pytest.mark.parametrize("shape,tile", GRIDS)
def test_outputs(shape, tile, kind, meth, f16):
    grid, cfg, rng, flags, bc = _case(shape, tile, meth, f16, kind)
    flags = np.where(flags & Flags.EXCLUDE, Flags.FLUID, flags).astype(np.uint8)
    f0 = initial_f(grid, cfg, rng)
    s = Solver(grid, cfg)
    rho = torch.empty(grid.num_points, device="cuda")
    u = torch.empty(grid.num_points * 2, device="cuda")
    q = torch.full((grid.num_points,), -7.0, device="cuda")
    fd, bcd, fld = to_dev(f0), to_dev(bc), to_dev(flags)
    s.compute_rho_u(rho, u, fd, bcd, fld, True)
    r_ref, u_ref = oracle.rho_u(cfg, grid, 32, f0, bc, flags, True)
    assert np.array_equal(rho.cpu().numpy().reshape(grid.shape), r_ref, equal_nan=True)
    assert np.array_equal(u.cpu().numpy().reshape((2,) + grid.shape), u_ref, equal_nan=True)
    s.q_criterion(q, fd, bcd, fld, u, 0.7, True)
    q_ref = oracle.q_criterion(cfg, grid, 32, f0, bc, flags, u_ref, 0.7, True, fill=-7.0)
    assert np.array_equal(q.cpu().numpy().reshape(grid.shape), q_ref, equal_nan=True)


@pytest.mark.parametrize("meth,f16,given", [("db", False, "u"), ("db", True, "rest"), ("eso", True, "rest")])
@pytest.mark.parametrize("shape,tile", GRIDS)
def test_initial_state(shape, tile, meth, f16, given):
    """(In place with a velocity, cells of several planes write one slot: at rest they agree.)"""
    grid, cfg, rng, _, _ = _case(shape, tile, meth, f16, "fluid")
    u = rng.normal(0, 0.03, (2,) + grid.shape).astype(np.float32) if given == "u" else None
    ref = np.zeros(grid.num_points * 9, oracle.f_dtype(cfg, 32))
    oracle.init(cfg, grid, 32, ref, 1.01, 0.7, u)
    fd = torch.zeros(ref.size, dtype=torch.int16 if f16 else torch.float32, device="cuda")
    Solver(grid, cfg).init_equilibrium(fd, 1.01, 0.7, None if u is None else torch.from_numpy(u).cuda())
    assert np.array_equal(fd.cpu().numpy().view(ref.dtype), ref)
