"""Two-sweep tile kernels of the multigrid V-cycle (GPU) against a V-cycle of SciPy matrices in FP64, on both sides of
the rule that keeps the couplings in shared memory (a launch of few tiles) or reads them through L1 (many tiles), and with
level tiles of other sizes than the framework's: any that fit the stages that two sweeps promise, and larger ones."""
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


def _compare(b, mg, rhs, specs, dtype):
    """The first PCG direction against the SciPy V-cycle of the systems of `specs` (the first ones of the batch)."""
    x, _ = _mg_solve(b, mg, rhs, iterations=1)
    sc = b._sim_cells.cpu().numpy()
    x, rhs = x.double().cpu().numpy(), rhs.double().cpu().numpy()
    tables = [t[0].cpu().numpy().reshape(-1, 12) for t in mg.levels_py]
    coefs = [(b.P.coef if l == 0 else mg.levels_py[l][2]).double().cpu().numpy().reshape(5, -1)
             for l in range(mg.num_levels)]
    nu = [2 if l >= mg.sub_level() else mg.levels[l].sweeps for l in range(mg.num_levels)]
    # rounding: in each level 5 applications of the stencil, each a chain of 7 operations; the sweeps do not amplify it
    # (damped Jacobi), so at most 5 * 7 roundings of the largest value a level
    bound = mg.num_levels * 5 * 7 * torch.finfo(dtype).eps / 2
    for k in range(len(specs)):
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
        print("%s system %d: %.2e (bound %.2e)" % (dtype, k, err, bound))
        assert err <= bound


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
    _compare(b, mg, rhs, specs[:4], dtype)


def _one_block(nx, ny, dtype):
    """Batch of one block of nx by ny square cells (a lid on one short side) after one step, its hierarchy, a seeded
    mean-free right-hand side."""
    from pict_b200.batch import BatchDomain
    from pict_b200.engine import PISOStepper
    from pict_b200.multigrid import hierarchy_for
    spec = dict(dims=2, viscosity=1e-3,
                blocks=[dict(coords=tensor_grid(np.linspace(0, nx / 100.0, nx + 1), np.linspace(0, ny / 100.0, ny + 1)))],
                ops=[("close", 0, f) for f in ("-x", "+x", "+y")] + [("close", 0, "-y", np.array([[1.0, 0.0]]))])
    b = BatchDomain([build_product(spec, dtype)], time_steps=[0.005])
    PISOStepper(b, time_step=0.005, advection_tol=1e-8, pressure_tol=1e-8).step()
    mg = hierarchy_for(b)
    mg.setup(b.P.coef, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    g = torch.Generator(device="cpu").manual_seed(12)
    rhs = torch.randn(b.getTotalSize(), generator=g, dtype=dtype).cuda()
    return spec, b, mg, rhs - rhs.mean()


def _retile(mg, tile):
    """The tile tables of the coarse levels cut into runs of `tile` cells."""
    from pict_b200.multigrid import level_tiles
    for l in range(1, mg.num_levels):
        table = mg.levels_py[l][0].cpu().numpy().reshape(-1, 12)
        t = torch.tensor(level_tiles(table[:, 0], table[:, 1] * table[:, 2], table[:, 7], tile), dtype=torch.int32, device="cuda")
        mg.levels[l].num_tiles, mg.levels[l].tiles = t.numel() // 4, t.data_ptr()
        mg.levels_py[l] = mg.levels_py[l][:3] + (t,)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tile", [100, 900, 4000])
def test_level_tiles_of_any_size(tile, dtype):
    """32 x 500 cells: level 1 is 16 x 250, whose tiles of 900 cells lie over at most 118 rows of 32 (3776 cells with the
    halo), more than the restriction's stage; a tile of 4000 cells is the whole level."""
    spec, b, mg, rhs = _one_block(32, 500, dtype)
    assert mg.levels[0].sweeps == 2 and mg.levels[1].sweeps == 2 and mg.sub_level() == 2
    _retile(mg, tile)
    _compare(b, mg, rhs, [spec], dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("announced", [700, 0, 10])
def test_rows_too_long_for_two_sweeps(announced, dtype):
    """1400 x 40 cells: rows of 700 on level 1 do not fit the stages.  Told to smooth that level twice, the solve smooths it
    once and converges, also where the level does not announce its rows; rows longer than announced are reported."""
    from pict_b200 import PISOtorch as P
    _, b, mg, rhs = _one_block(1400, 40, dtype)
    assert mg.levels[1].max_block_sx == 700 and mg.levels[1].sweeps == 1 and mg.sub_level() > 1
    mg.levels[1].sweeps = 2
    mg.levels[1].max_block_sx = announced
    tol = 1e-4 if dtype == torch.float32 else 1e-10
    x = torch.zeros_like(rhs)
    info = torch.zeros(24, dtype=torch.uint8, device="cuda")
    ws = torch.full((mg.workspace_bytes(b._desc),), 255, dtype=torch.uint8, device="cuda")   # NaN where nothing writes
    mg.solve(b._desc, rhs, x, 100, tol, info, ws, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    (i,) = P.decode_infos(info)
    if announced == 10:
        assert i.status == 1 and not i.converged, i
        return
    assert i.converged and i.status == 0, i
    A = _stencil_matrix(b.P.coef.double().cpu().numpy(), [[0, 1400, 40, 1, 0, 0, 0]], 2)
    r = rhs.double().cpu().numpy() - A @ x.double().cpu().numpy()
    # the recursion's residual plus the rounding of its at most 100 updates at the largest row sum and iterate
    drift = 100 * torch.finfo(dtype).eps * abs(A).sum(axis=1).max() * float(x.abs().max())
    assert np.sqrt((r ** 2).mean()) <= tol + drift


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("copies", [0, 140])
def test_couplings_across_fixed_faces_are_not_read(copies, dtype):
    """A face without a neighbour has no term, whatever its coefficient holds: NaN there changes no bit of the solution."""
    from pict_b200.batch import BatchDomain
    from pict_b200.engine import PISOStepper
    from pict_b200.multigrid import hierarchy_for
    specs = [lid_cavity(100, viscosity=1e-3), lid_cavity(37, viscosity=1e-3), _channel(64, 48)]
    specs += [specs[0]] * copies
    b = BatchDomain([build_product(s, dtype) for s in specs], time_steps=[0.005] * len(specs))
    PISOStepper(b, time_step=0.005, advection_tol=1e-8, pressure_tol=1e-8).step()
    mg = hierarchy_for(b)
    assert mg.levels[0].sweeps == 2
    g = torch.Generator(device="cpu").manual_seed(13)
    rhs = torch.randn(b.getTotalSize(), generator=g, dtype=dtype).cuda()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = []
    for poison in (False, True):
        coef = b.P.coef.clone().reshape(5, -1)
        if poison:
            coef[1:][b._nbr.reshape(4, -1) < 0] = float("nan")
        mg.setup(coef, st)
        out.append(_mg_solve(b, mg, rhs, iterations=3)[0])
    assert bool(torch.isfinite(out[0]).all()) and torch.equal(out[0], out[1])
