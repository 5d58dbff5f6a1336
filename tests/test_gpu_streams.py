"""One solver stepped on two streams without waiting in between: calls that run while a long run of the
other stream is in flight, directly or from a captured graph, keep their own boundary values (and on the
generic kernel their own flags), and give the words of the same steps taken one by one."""
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

DELAY = 2_000_000  # clock cycles that the second stream waits before its steps: about a millisecond


@pytest.mark.parametrize("how", ["run", "steps", "captured"])
@pytest.mark.parametrize("lat,shape,tile,path", [("D2Q9", (64, 96, 1), (16, 16, 1), 0), ("D3Q19", (32, 32, 24), (8, 8, 4), 0),
                                                 ("D3Q19", (32, 32, 24), (8, 8, 4), 1), ("D3Q19", (41, 29, 17), "untiled", 0)])
def test_overlapping_streams(lat, shape, tile, path, how):
    grid = make_grid(lat, shape, tile)
    cfg = LBM_Config(LBM_method.DOUBLE_BUFFER, BCs={Flags.EQUILIBRIUM})
    rng = np.random.default_rng(grid.num_points)
    one, ref = Solver(grid, cfg), Solver(grid, cfg)
    for s in (one, ref):
        s.set_kernel_path(path)
    flags, _ = mixed_flags(grid, rng)
    side = []  # per stream: its stream, buffers, boundary values and flags
    for k in range(2):
        if one.kernel_path == 1 and k == 1:
            flags, _ = mixed_flags(grid, rng)
        f0 = initial_f(grid, cfg, rng)
        side.append(dict(stream=torch.cuda.Stream(), f=[to_dev(f0) for _ in range(4)], fl=to_dev(flags),
                         bc=to_dev(_bc(grid, rng, 0.9 - 0.7 * k))))
    A, B = side

    def run(d, n):
        one.run(d["f"][0], d["f"][1], d["bc"], d["fl"], 0.8, n, 0, d["stream"])

    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    run(A, 2)
    run(A, 64)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=B["stream"]):
        run(B, 20)
    torch.cuda.synchronize()
    for _ in range(3):  # B's steps run after A's run has been taken up, and A's next run while B's steps do
        with torch.cuda.stream(B["stream"]):
            torch.cuda._sleep(DELAY)
            if how == "captured":
                graph.replay()
        if how == "run":
            run(B, 20)
        elif how == "steps":
            for _ in range(10):
                run(B, 2)
        run(A, 64)
        run(A, 64)
        torch.cuda.synchronize()
    for d, n in ((A, 66 + 3 * 128), (B, 60)):
        _one_by_one(ref, cfg, d["f"][2], d["f"][3], d["bc"], d["fl"], 0.8, n)
        torch.cuda.synchronize()
        for k in (0, 1):
            assert torch.equal(d["f"][k].view(torch.int32), d["f"][2 + k].view(torch.int32))
