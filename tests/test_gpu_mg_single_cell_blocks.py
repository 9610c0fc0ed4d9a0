"""Blocks that reach one cell before the coarsest level (GPU): a small cavity beside a large one is coarsened as often as
the large one, so its block has one cell on several levels.  The operator of such a block is 0 up to rounding; it is not
smoothed, and the small system converges like it does alone."""
import ctypes

import numpy as np
import pytest
import torch

from setups import build_product, lid_cavity

pytestmark = pytest.mark.gpu


def _used(sides, seed, dtype, reduction):
    """PCG iterations that each cavity needs to reduce a random right-hand side by `reduction` (cap 40)."""
    from pict_b200 import PISOtorch as P
    from pict_b200.batch import BatchDomain
    from pict_b200.engine import PISOStepper
    from pict_b200.multigrid import hierarchy_for
    b = BatchDomain([build_product(lid_cavity(n, viscosity=1e-3), dtype) for n in sides],
                    time_steps=[0.5 / n for n in sides], order="given")
    PISOStepper(b, time_step=0.01, advection_tol=1e-7, pressure_tol=1e-7).step()
    mg = hierarchy_for(b)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    mg.setup(b.P.coef, st)
    g = torch.Generator(device="cpu").manual_seed(seed)
    sc = b._sim_cells.cpu().numpy()
    rhs = torch.empty(b.getTotalSize(), dtype=torch.float64)
    for s0, s1 in zip(sc[:-1], sc[1:]):
        r = torch.randn(int(s1 - s0), generator=g, dtype=torch.float64)
        r -= r.mean()
        rhs[s0:s1] = r / r.norm() * np.sqrt(s1 - s0)   # RMS 1 in every system
    rhs = rhs.to("cuda", dtype)
    x = torch.zeros_like(rhs)
    info = torch.zeros(b.num_sims * 24, dtype=torch.uint8, device="cuda")
    ws = torch.empty(mg.workspace_bytes(b._desc), dtype=torch.uint8, device="cuda")
    mg.solve(b._desc, rhs, x, 40, reduction, info, ws, st)
    return mg, P.decode_infos(info)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("sides", [(256, 32, 28, 24, 20, 16, 9, 5), (256, 6, 4, 3), (200, 32), (130, 17, 8)], ids=str)
def test_small_systems_beside_large_ones_converge(sides, dtype):
    # Only the systems whose block has one cell on a level that is not the coarsest.  Their FP32 solves come to 1e-7 and
    # lower (the rounding of A p, whose mean a singular solve cannot reduce; for sides above 64 it is 1e-8 to 2e-6, with one
    # smoothing sweep and with two alike); smoothed one-cell blocks left 1e-5 to 1e-4.
    reduction = 1e-6 if dtype == torch.float32 else 1e-12
    for seed in range(4):
        mg, infos = _used(sides, seed, dtype, reduction)
        small = [i for n, i in zip(sides, infos) if n <= 2 ** (mg.num_levels - 2)]
        assert len(small) >= 1
        assert all(i.converged and i.isFiniteResidual and i.status == 0 for i in small), (sides, infos)
