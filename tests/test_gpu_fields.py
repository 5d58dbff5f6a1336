"""The kernels between the lattice and the row-major fields (lbm_fields.cuh), against the oracle bit
for bit, at the sizes where their bricks of 32 lanes x 32 planes have remainders: extents around a
brick's along every axis, tile rows shorter and longer than a warp, the untiled layout, and domains
with walls, mixed flags or none (a brick without any flag takes the form that gathers none)."""
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

# lattice, shape, tile
GRIDS = [("D3Q19", (33, 5, 35), "untiled"), ("D3Q19", (8, 4, 32), (8, 4, 4)), ("D3Q19", (10, 9, 31), (2, 3, 1)),
         ("D3Q19", (40, 6, 3), (40, 2, 3)), ("D3Q27", (16, 8, 36), (16, 4, 4)), ("D3Q27", (3, 34, 65), (1, 1, 1)),
         ("D2Q9", (33, 34, 1), "untiled"), ("D2Q9", (48, 80, 1), (16, 16, 1)), ("D2Q9", (9, 130, 1), (3, 2, 1)),
         ("D2Q9", (2, 1030, 1), (1, 1, 1)),
         ("D3Q19", (97, 83, 81), "untiled"), ("D2Q9", (800, 816, 1), (16, 16, 1))]


def _flags(grid, kind, rng):
    flags, bc = mixed_flags(grid, rng)
    if kind == "fluid":
        flags[:] = 0
    elif kind == "sparse":  # most bricks without a flag
        flags[rng.random(flags.size) < 0.999] = 0
    else:
        flags = np.where(flags & Flags.EXCLUDE, Flags.FLUID, flags).astype(np.uint8)
    return flags, bc


@pytest.mark.parametrize("meth,f16", [("db", False), ("eso", True)])
@pytest.mark.parametrize("kind", ["fluid", "sparse", "mixed"])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_outputs_at_brick_edges(lat, shape, tile, kind, meth, f16):
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(len(kind) + grid.num_points)
    flags, bc = _flags(grid, kind, rng)
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

