"""The kernels between the lattice and the row-major fields (lbm_fields.cuh), against the oracle bit
for bit, at the sizes where their bricks of 32 lanes x 32 planes have remainders: extents around a
brick's along every axis, tile rows shorter and longer than a warp, the untiled layout, and domains
with walls, mixed flags or none (a brick without any flag takes the form that gathers none); the
Float16C codec over arrays, and the mass and momentum sums."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method, _capi
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


@pytest.mark.parametrize("meth,f16,given", [("db", False, "u+grad"), ("eso", True, "u+grad"), ("eso", False, "grad"),
                                            ("db", True, "u"), ("db", False, "rest")])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_init_at_brick_edges(lat, shape, tile, meth, f16, given):
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points)
    u = rng.normal(0, 0.03, (grid.D,) + grid.shape).astype(np.float32) if "u" in given else None
    g = rng.normal(0, 1e-3, (grid.D * grid.D,) + grid.shape).astype(np.float32) if "grad" in given else None
    ref = np.zeros(grid.num_points * grid.Q, oracle.f_dtype(cfg, 32))
    oracle.init(cfg, grid, 32, ref, 1.01, 0.7, u, g)
    fd = torch.zeros(ref.size, dtype=torch.int16 if f16 else torch.float32, device="cuda")
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()  # noqa: E731
    Solver(grid, cfg).init_equilibrium(fd, 1.01, 0.7, dev(u), dev(g))
    assert np.array_equal(fd.cpu().numpy().view(ref.dtype), ref)


@pytest.mark.parametrize("n", [1, 7, 8, 4096, 4096 * 3 + 5])
@pytest.mark.parametrize("shift", [0, 1, 8])
def test_codec_words_and_remainders(n, shift):
    """The codec by whole 16-byte words, its remainder and arrays that are not 16-byte aligned."""
    rng = np.random.default_rng(n)
    x = np.concatenate([rng.normal(0, 1, n), rng.normal(0, 1e-6, n)]).astype(np.float32)[rng.permutation(2 * n)[:n]]
    want = oracle.f16c_encode(x)
    src = torch.zeros(n + shift, device="cuda")[shift:]
    src.copy_(torch.from_numpy(x))
    out = torch.zeros(n + shift + 1, dtype=torch.int16, device="cuda")
    code = out[shift:shift + n]
    _capi.check(_capi.lib().lbm_float16c_encode(src.data_ptr(), code.data_ptr(), n, None))
    assert np.array_equal(code.cpu().numpy().view(np.uint16), want)
    assert int(out[shift + n]) == 0  # nothing past the end
    back = torch.zeros(n + shift + 1, device="cuda")
    _capi.check(_capi.lib().lbm_float16c_decode(code.data_ptr(), back[shift:].data_ptr(), n, None))
    assert np.array_equal(back[shift:shift + n].cpu().numpy().view(np.uint32), oracle.f16c_decode(want).view(np.uint32))
    assert float(back[shift + n]) == 0.0


@pytest.mark.parametrize("scale", ["flow", "tiny", "huge", "mixed"])
@pytest.mark.parametrize("lat,meth,ddf", [("D2Q9", "db", False), ("D3Q19", "db", True), ("D3Q27", "eso", True)])
def test_mass_momentum_sums(lat, meth, ddf, scale):
    """The reduction's split sums against a float64 sum of the same populations: ordinary cells, cells
    too small or too large for the split (added in float64) and both in one domain.  Float64
    summation bounds both errors by 2^-53 times the terms of a cell and of the reduction tree
    (below 2^10 of them) relative to the sum of magnitudes."""
    shape = {"D2Q9": (48, 34, 1), "D3Q19": (20, 18, 16), "D3Q27": (12, 10, 9)}[lat]
    grid = make_grid(lat, shape, "untiled")
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, DDF_shift=ddf)
    rng = np.random.default_rng(11)
    f = initial_f(grid, cfg, rng).reshape(grid.Q, -1)
    if scale == "tiny":
        f *= np.float32(2.0 ** -40)
    elif scale == "huge":
        f *= np.float32(1e30)
    elif scale == "mixed":
        f *= np.float32(2.0) ** rng.integers(-60, 12, f.shape[1]).astype(np.float32)
        f[:, rng.random(f.shape[1]) < 0.2] = 0.0
    f = np.ascontiguousarray(f).reshape(-1)
    nat = grid.layouts.from_layout(f, grid.Q).transpose(3, 0, 1, 2).astype(np.float64)
    g = nat.copy()
    if meth == "eso":  # after an odd step: f[pos] was stored at x + c in slot pos, f[neg] at x in slot neg
        for p in range(1, grid.Q, 2):
            c = [int(v) for v in grid.lattice.directions[p]]
            g[p] = np.roll(nat[p], [-v for v in c[:grid.D]], axis=tuple(range(grid.D)))
    want = [g.sum() + (grid.num_points if ddf else 0)]
    size = [np.abs(g).sum() + (grid.num_points if ddf else 0)]
    for d in range(grid.D):
        c = grid.lattice.directions[:, d].astype(np.float64)
        want.append((g * c[:, None, None, None]).sum())
        size.append(np.abs(g * c[:, None, None, None]).sum())
    flags = torch.zeros(grid.num_points, dtype=torch.uint8, device="cuda")
    got = Solver(grid, cfg).mass_momentum(to_dev(f), flags, after_odd_step=True)
    for k in range(grid.D + 1):
        assert abs(got[k] - want[k]) <= 2.0 ** -43 * size[k], (k, got[k], want[k])
