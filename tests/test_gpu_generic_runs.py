"""The generic kernel in runs long enough for its masks, in turn with calls that gather the neighbours'
flags: flags rewritten between calls, in buffers with and without 16-byte alignment, give the words of the
same steps taken one by one; and a grid large enough that a single step uses the masks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev
from tests.test_gpu_walls import _bc, _one_by_one

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("meth,f16,coll,les", [("db", False, "SRT", False), ("eso", True, "TRT", True),
                                               ("db", True, "RLBM", True), ("eso", False, "KBC", False)])
@pytest.mark.parametrize("lat,shape,tile", [("D3Q19", (33, 5, 7), "untiled"), ("D3Q19", (31, 2, 9), (31, 1, 3)),
                                            ("D3Q27", (6, 10, 5), (3, 5, 5)), ("D2Q9", (67, 13, 1), "untiled"),
                                            ("D2Q9", (30, 9, 1), (5, 3, 1)), ("D3Q19", (16, 16, 8), (8, 8, 4))])
def test_runs_follow_the_flags(lat, shape, tile, meth, f16, coll, les):
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, collision_op=coll, LES=les, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points + len(coll))
    mixed, _ = mixed_flags(grid, rng)
    sparse = np.where(rng.random(mixed.size) < 0.01, mixed, 0).astype(np.uint8)
    N = grid.num_points
    fl = torch.zeros(N + 1, dtype=torch.uint8, device="cuda")
    views = [fl[:N], fl[1:]]  # the second is not aligned
    run, ref = Solver(grid, cfg), Solver(grid, cfg)
    for s in (run, ref):
        s.set_kernel_path(1)
    f0 = initial_f(grid, cfg, rng)
    a1, b1, a2, b2 = (to_dev(f0) for _ in range(4))
    bc = to_dev(_bc(grid, rng, 0.5))
    word = torch.int16 if f16 else torch.int32
    for k, (n, flags) in enumerate([(16, np.zeros_like(mixed)), (16, sparse), (2, mixed), (40, mixed), (16, sparse),
                                    (2, np.zeros_like(mixed)), (16, sparse), (64, mixed), (16, np.zeros_like(mixed))]):
        v = views[k % 2]
        v.copy_(torch.from_numpy(flags))
        bc.copy_(torch.from_numpy(_bc(grid, rng, 0.5)))
        run.run(a1, b1, bc, v, 0.8, n, 0)
        _one_by_one(ref, cfg, a2, b2, bc, v, 0.8, n)
        assert torch.equal(a1.view(word), a2.view(word)) and torch.equal(b1.view(word), b2.view(word)), f"part {k}"


@pytest.mark.parametrize("lat,shape", [("D2Q9", (2053, 2047, 1)), ("D3Q19", (131, 129, 127))])
def test_single_steps_with_masks(lat, shape):
    """Single steps on the owner's stream (masks) and on another one (gathered flags) agree."""
    grid = make_grid(lat, shape, "untiled")
    cfg = LBM_Config(LBM_method.DOUBLE_BUFFER, BCs={Flags.EQUILIBRIUM})
    rng = np.random.default_rng(5)
    s = Solver(grid, cfg)
    N = grid.num_points
    gen = torch.Generator(device="cuda").manual_seed(1)
    f = torch.zeros(N * grid.Q, device="cuda")
    s.init_equilibrium(f, 1.0, 0.8)
    f *= 1 + 0.01 * torch.rand(f.shape, device="cuda", generator=gen)
    bc = to_dev(_bc(grid, rng, 0.5))
    other, out, gathered = torch.cuda.Stream(), torch.zeros_like(f), torch.zeros_like(f)
    for share in (0.0, 1e-4, 0.05):
        flags = (torch.rand(N, device="cuda", generator=gen) < share).to(torch.uint8) * Flags.SOLID
        s.double_buffer_step(out, f, bc, flags, 0.8)
        torch.cuda.synchronize()
        s.double_buffer_step(gathered, f, bc, flags, 0.8, other)
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), gathered.view(torch.int32)), share
