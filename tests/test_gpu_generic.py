"""The generic step kernel (any tile, any size) against the oracle, bit for bit, where its warp masks
and offsets can go wrong: extents that are no multiple of a warp, rows shorter and longer than one, the
untiled layout, isolated flags, flags that change between calls or are not 16-byte aligned, and a
lattice of more than 2^31 elements (64-bit offsets; also the initial state and the outputs)."""
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

GRIDS = [("D3Q19", (33, 5, 7), "untiled"), ("D3Q19", (31, 2, 9), (31, 1, 3)), ("D3Q27", (6, 10, 5), (3, 5, 5)),
         ("D2Q9", (67, 13, 1), "untiled"), ("D2Q9", (30, 9, 1), (5, 3, 1)), ("D3Q19", (16, 16, 8), (8, 8, 4))]


def _steps(s, cfg, meth, a, b, bc, fl, tau, k):
    if meth == "eso":
        s.esoteric_pull_step(a, bc, fl, tau, k % 2 == 0)
        return a, a
    s.double_buffer_step(b, a, bc, fl, tau)
    return b, a


@pytest.mark.parametrize("meth,f16,coll,les", [("db", False, "SRT", False), ("eso", True, "TRT", True),
                                               ("db", True, "RLBM", True), ("eso", False, "KBC", False)])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_generic_masks_follow_the_flags(lat, shape, tile, meth, f16, coll, les):
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, collision_op=coll, LES=les, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points + len(coll))
    mixed, bc = mixed_flags(grid, rng)
    bc = np.nan_to_num(bc, nan=0.01)
    sparse = np.where(rng.random(mixed.size) < 0.01, mixed, 0).astype(np.uint8)
    N = grid.num_points
    fl = torch.zeros(N + 1, dtype=torch.uint8, device="cuda")
    views = [fl[:N], fl[1:]]  # the second is not aligned
    s = Solver(grid, cfg)
    s.set_kernel_path(1)
    f = initial_f(grid, cfg, rng)
    f2 = f.copy()
    a, b = to_dev(f), to_dev(f)
    bcd = to_dev(bc)
    tau = 0.8
    for k, flags in enumerate([np.zeros_like(mixed), sparse, sparse, mixed, np.zeros_like(mixed), sparse]):
        v = views[k % 2]
        v.copy_(torch.from_numpy(flags))
        a, b = _steps(s, cfg, meth, a, b, bcd, v, tau, k)
        if meth == "eso":
            oracle.step(cfg, grid, 32, f, f, bc, flags, tau, k % 2 == 0)
        else:
            oracle.step(cfg, grid, 32, f2, f, bc, flags, tau)
            f, f2 = f2, f
        got = a.cpu().numpy().view(np.uint16 if f16 else np.uint32)
        assert np.array_equal(got, f.view(np.uint16 if f16 else np.uint32)), f"step {k}"


@pytest.mark.parametrize("meth", ["db", "eso"])
def test_more_than_2_31_elements(meth):
    """A periodic domain whose state repeats: every copy of the small domain in the large one (2.2e9
    codes) holds the small domain's words."""
    small, reps = (24, 18, 20), (18, 24, 22)
    gs = make_grid("D3Q27", small, "untiled")
    gb = make_grid("D3Q27", tuple(a * b for a, b in zip(small, reps)), "untiled")
    assert gb.num_points * 27 > 2 ** 31
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, DDF_shift=True, use_float16c=True, include_moving_boundary=False)
    rng = np.random.default_rng(3)
    u = rng.normal(0, 0.02, (3,) + small).astype(np.float32)
    us = torch.from_numpy(u).cuda()
    out = []
    for g, ud in ((gs, us), (gb, us.repeat(1, *reps).contiguous())):
        s = Solver(g, cfg)
        fa = torch.empty(g.num_points * 27, dtype=torch.int16, device="cuda")
        s.init_equilibrium(fa, 1.0, 0.7, ud)
        del ud
        fb = torch.zeros_like(fa) if meth == "db" else None
        fl = torch.zeros(g.num_points, dtype=torch.uint8, device="cuda")
        bc = torch.zeros(g.num_points * 4, device="cuda")
        s.run(fa, fb, bc, fl, 0.7, 2, 0)
        rho, v = torch.empty(g.shape, device="cuda"), torch.empty((3,) + g.shape, device="cuda")
        s.compute_rho_u(rho, v, fa, bc, fl, True)
        out.append((fa.view(27, g.nz, g.ny, g.nx), rho, v))
        s.close()
    ref = np.zeros(gs.num_points * 27, np.uint16)
    oracle.init(cfg, gs, 32, ref, 1.0, 0.7, u)
    f2, fl, bc = ref.copy(), np.zeros(gs.num_points, np.uint8), np.zeros(gs.num_points * 4, np.float32)
    for k in range(2):
        oracle.step(cfg, gs, 32, ref if meth == "eso" else f2, ref, bc, fl, 0.7, k % 2 == 0)
        if meth == "db":
            ref, f2 = f2, ref
    (fs, rs, vs), (fb, rb, vb) = out
    assert np.array_equal(fs.cpu().numpy().view(np.uint16).ravel(), ref)
    for q in range(27):
        assert torch.equal(fb[q], fs[q].repeat(reps[2], reps[1], reps[0])), q
    assert torch.equal(rb, rs.repeat(*reps))
    for d in range(3):
        assert torch.equal(vb[d], vs[d].repeat(*reps))
