"""The two forms of the kernels between the lattice and the row-major fields, bricks and one thread per cell
(by_cell in lbm_fields.cuh), against the oracle bit for bit: grids large enough for bricks of 8 and of 32
planes with remainders along every axis and around the lines of the rule, thin grids, and tiles whose runs
along a warp are short."""
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

GRIDS = [  # bricks of 8 planes
    ("D3Q19", (33, 65, 35), "untiled"), ("D3Q19", (10, 63, 120), (2, 3, 1)), ("D3Q19", (40, 46, 39), (40, 2, 3)),
    ("D3Q27", (48, 40, 36), (16, 4, 4)), ("D3Q27", (4, 170, 130), (4, 5, 1)), ("D3Q19", (150, 90, 5), "untiled"),
    ("D2Q9", (330, 200, 1), "untiled"), ("D2Q9", (272, 256, 1), (16, 16, 1)), ("D2Q9", (9, 7302, 1), (3, 2, 1)),
    # bricks of 32 planes
    ("D3Q19", (10, 251, 260), (2, 1, 13)), ("D3Q19", (271, 267, 9), "untiled"), ("D2Q9", (9, 70001, 1), "untiled"),
    # one thread per cell
    ("D3Q19", (33, 5, 35), "untiled"), ("D2Q9", (33, 34, 1), "untiled"), ("D3Q19", (150, 150, 4), "untiled"),
    ("D3Q27", (130, 258, 2), (2, 3, 1)), ("D2Q9", (33001, 5, 1), "untiled"), ("D2Q9", (2, 33000, 1), (1, 1, 1)),
    ("D3Q19", (41, 42, 43), (1, 1, 1)), ("D3Q19", (42, 41, 40), (2, 1, 1)), ("D3Q19", (42, 40, 44), (2, 2, 2))]


def _cfg(meth, f16):
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    return LBM_Config(m, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)


@pytest.mark.parametrize("meth,f16", [("db", False), ("eso", True)])
@pytest.mark.parametrize("kind", ["fluid", "mixed"])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_outputs(lat, shape, tile, kind, meth, f16):
    grid, cfg = make_grid(lat, shape, tile), _cfg(meth, f16)
    rng = np.random.default_rng(grid.num_points)
    flags, bc = mixed_flags(grid, rng)
    flags = np.where(flags & Flags.EXCLUDE, Flags.FLUID, flags).astype(np.uint8) if kind == "mixed" else np.zeros_like(flags)
    f0 = initial_f(grid, cfg, rng)
    s = Solver(grid, cfg)
    rho = torch.empty(grid.num_points, device="cuda")
    u = torch.empty(grid.num_points * grid.D, device="cuda")
    q = torch.full((grid.num_points,), -7.0, device="cuda")
    fd, bcd, fld = to_dev(f0), to_dev(bc), to_dev(flags)
    s.compute_rho_u(rho, u, fd, bcd, fld, True)
    r_ref, u_ref = oracle.rho_u(cfg, grid, 32, f0, bc, flags, True)
    assert np.array_equal(rho.cpu().numpy().reshape(grid.shape), r_ref, equal_nan=True)
    assert np.array_equal(u.cpu().numpy().reshape((grid.D,) + grid.shape), u_ref, equal_nan=True)
    s.q_criterion(q, fd, bcd, fld, u, 0.7, True)
    q_ref = oracle.q_criterion(cfg, grid, 32, f0, bc, flags, u_ref, 0.7, True, fill=-7.0)
    assert np.array_equal(q.cpu().numpy().reshape(grid.shape), q_ref, equal_nan=True)


@pytest.mark.parametrize("meth,f16,given", [("db", False, "u+grad"), ("eso", True, "u+grad"), ("eso", False, "grad"),
                                            ("db", True, "u"), ("db", False, "rest")])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_initial_state(lat, shape, tile, meth, f16, given):
    grid, cfg = make_grid(lat, shape, tile), _cfg(meth, f16)
    rng = np.random.default_rng(grid.num_points)
    u = rng.normal(0, 0.03, (grid.D,) + grid.shape).astype(np.float32) if "u" in given else None
    g = rng.normal(0, 1e-3, (grid.D * grid.D,) + grid.shape).astype(np.float32) if "grad" in given else None
    ref = np.zeros(grid.num_points * grid.Q, oracle.f_dtype(cfg, 32))
    oracle.init(cfg, grid, 32, ref, 1.01, 0.7, u, g)
    fd = torch.zeros(ref.size, dtype=torch.int16 if f16 else torch.float32, device="cuda")
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()  # noqa: E731
    Solver(grid, cfg).init_equilibrium(fd, 1.01, 0.7, dev(u), dev(g))
    assert np.array_equal(fd.cpu().numpy().view(ref.dtype), ref)
