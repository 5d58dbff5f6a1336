"""Large double-buffer batches (two cells per thread) against the single-domain steps.  The batched step
always computes the exact arithmetic."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.batch import BatchSolver
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu

# (lattice, domain shapes, tile): units at the first batch that steps two cells per thread (1,216), one
# below it, a remainder of the 4 units of a CTA, and tiles one cell wide, which never do
DOMAINS = [("D3Q19", [(80, 80, 48), (8, 8, 4), (24, 8, 20)], (8, 8, 4)),
           ("D3Q19", [(80, 80, 48), (24, 8, 20)], (8, 8, 4)),
           ("D2Q9", [(512, 504, 1), (32, 8, 1), (96, 648, 1)], (32, 8, 1)),
           ("D3Q19", [(16, 160, 192), (7, 32, 16)], (1, 16, 16))]


@pytest.mark.parametrize("lat,shapes,tile", DOMAINS)
@pytest.mark.parametrize("store,coll,les", [("fp32", "SRT", False), ("f16c", "TRT", True), ("fp32", "RLBM", False),
                                            ("f16c", "KBC", False)])
def test_large_batch_equals_single_domain_steps(lat, shapes, tile, store, coll, les):
    """Populations equal those of each domain stepped alone, word for word, in replayed and single steps,
    with buffers that are 8-byte aligned, then set again to ones that are not, then back."""
    rng = np.random.default_rng(11)
    f16 = store == "f16c"
    cfg = LBM_Config(LBM_method.DOUBLE_BUFFER, collision_op=coll, LES=les, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16,
                     use_float16c=f16)
    grids = [make_grid(lat, s, tile) for s in shapes]
    batch = BatchSolver(grids, cfg)
    bufs, ref = [], []
    for g in grids:
        flags, bc = mixed_flags(g, rng)
        flags[rng.random(flags.size) < 0.97] = 0
        f0 = to_dev(initial_f(g, cfg, rng))
        pads = [torch.zeros(f0.numel() + 1, dtype=f0.dtype, device="cuda") for _ in range(2)]
        bufs.append((pads, to_dev(np.nan_to_num(bc, nan=0.01)), to_dev(flags)))
        ref.append([f0.clone(), f0.clone()])
    word = torch.int16 if f16 else torch.int32
    solvers = [Solver(g, cfg) for g in grids]
    k = 0
    for shift, n in ((0, 66), (1, 65), (0, 2)):
        views = []
        for i, (pads, bc, fl) in enumerate(bufs):
            v = [p[shift:shift + ref[i][0].numel()] for p in pads]
            for a, b in zip(v, ref[i]):
                a.copy_(b)
            views.append(v)
            batch.set_domain(i, v[0], v[1], bc, fl, 0.6)
        batch.run(n, k)
        for i, (_, bc, fl) in enumerate(bufs):
            for j in range(n):
                p = (k + j) % 2
                solvers[i].double_buffer_step(ref[i][1 - p], ref[i][p], bc, fl, 0.6)
        k += n
        for i, v in enumerate(views):
            assert torch.equal(v[0].view(word), ref[i][0].view(word)), f"domain {i} lattice A differs"
            assert torch.equal(v[1].view(word), ref[i][1].view(word)), f"domain {i} lattice B differs"
