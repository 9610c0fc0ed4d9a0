"""Two-sweep tile kernels of the multigrid V-cycle (GPU) against a V-cycle of SciPy matrices in FP64, on both sides of
the rule that keeps the couplings in shared memory (a launch of few tiles) or reads them through L1 (many tiles)."""
import ctypes

import numpy as np
import pytest
import torch

from setups import build_product, lid_cavity, stretched, tensor_grid
from test_gpu_multigrid import _aggregation, _mg_solve, _stencil_matrix

pytestmark = pytest.mark.gpu

OMEGA, SCALE, COARSE_SWEEPS = 0.8, 2.0, 8    # the defaults of MGHierarchy.solve


def _channel(nx, ny):
    """x-periodic block, stretched in y (halved in y first)."""
    return dict(dims=2, viscosity=1e-2,
                blocks=[dict(coords=tensor_grid(np.linspace(0, 2.0, nx + 1), stretched(ny, length=1.0, beta=2.0)))],
                ops=[("periodic", 0, "x"), ("close", 0, "-y"), ("close", 0, "+y")])


def _vcycle(A, R, nu, b, l=0):
    d = A[l].diagonal()

    def sweeps(x, n):
        for _ in range(n):
            x = x + OMEGA * (b - A[l] @ x) / d
        return x
    if l == len(A) - 1:
        x = sweeps(np.zeros_like(b), COARSE_SWEEPS)
        return x - x.mean()
    x = sweeps(np.zeros_like(b), nu[l])
    e = _vcycle(A, R, nu, R[l] @ (b - A[l] @ x), l + 1)
    return sweeps(x + SCALE * (R[l].T @ e), nu[l])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("copies", [0, 140])
def test_vcycle_matches_scipy(copies, dtype):
    """The first PCG direction is the V-cycle of the right-hand side (up to a factor and its mean).  Widths that the
    tiles cut mid-row, x-periodic rows, odd sides and per-block coarsening; with 140 copies of the 100^2 block every
    finest launch has more than 4 tiles an SM."""
    from pict_b200.batch import BatchDomain
    from pict_b200.engine import PISOStepper
    from pict_b200.multigrid import hierarchy_for
    specs = [lid_cavity(100, viscosity=1e-3), lid_cavity(37, viscosity=1e-3), _channel(64, 48), _channel(33, 21)]
    specs += [specs[0]] * copies
    b = BatchDomain([build_product(s, dtype) for s in specs], time_steps=[0.005] * len(specs))
    PISOStepper(b, time_step=0.005, advection_tol=1e-8, pressure_tol=1e-8).step()
    mg = hierarchy_for(b)
    assert mg.levels[0].sweeps == 2
    mg.setup(b.P.coef, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    g = torch.Generator(device="cpu").manual_seed(11)
    rhs = torch.randn(b.getTotalSize(), generator=g, dtype=dtype).cuda()
    sc = b._sim_cells.cpu().numpy()
    for k in range(len(specs)):
        rhs[sc[k]:sc[k + 1]] -= rhs[sc[k]:sc[k + 1]].mean()
    x, _ = _mg_solve(b, mg, rhs, iterations=1)
    x, rhs = x.double().cpu().numpy(), rhs.double().cpu().numpy()
    tables = [t[0].cpu().numpy().reshape(-1, 12) for t in mg.levels_py]
    coefs = [(b.P.coef if l == 0 else mg.levels_py[l][2]).double().cpu().numpy().reshape(5, -1)
             for l in range(mg.num_levels)]
    nu = [2 if l >= mg.sub_level() else mg.levels[l].sweeps for l in range(mg.num_levels)]
    # rounding: at most 7 levels, in each 5 applications of the stencil, each a chain of 7 operations; the sweeps do
    # not amplify it (damped Jacobi), so at most 7 * 5 * 7 roundings of the largest value
    assert mg.num_levels <= 7
    bound = 7 * 5 * 7 * torch.finfo(dtype).eps / 2
    for k in range(4):
        A, R, prev = [], [], None
        for table, coef in zip(tables, coefs):
            row = table[k].copy()
            n = int(row[1]) * int(row[2])
            off = int(row[0])
            row[0] = 0
            A.append(_stencil_matrix(coef[:, off:off + n].reshape(-1), [row], 2))
            if prev is not None:
                R.append(_aggregation([prev], [row]))
            prev = row
        z = _vcycle(A, R, nu, rhs[sc[k]:sc[k + 1]])
        z -= z.mean()
        xk = x[sc[k]:sc[k + 1]]
        err = np.abs(xk * (z @ z) / (xk @ z) - z).max() / np.abs(z).max()
        print("%s copies %d system %d: %.2e (bound %.2e)" % (dtype, copies, k, err, bound))
        assert err <= bound
