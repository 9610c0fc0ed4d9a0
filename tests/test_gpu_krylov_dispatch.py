"""Which kernel solves a domain, and what that changes (GPU): the limits of the on-chip and the cluster solves, and a
system's result alone, in batches that are solved alike and in batches that are not."""
import ctypes

import numpy as np
import pytest
import torch

from setups import build_product
from test_gpu_resident_krylov import _box, _matrix

pytestmark = pytest.mark.gpu

SMALL = [(20, 20), (33, 17), (48, 31), (17, 40), (64, 64), (10, 12), (25, 25), (91, 30)]


KRYLOV = ("k_cg1_resident", "k_cg1_cluster", "k_cg1<", "k_bicgstab_resident", "k_bicgstab<")


def _kernels(fn):
    """The Krylov kernels that fn launches (run again where the profiler has lost its records, which it does at times)."""
    from torch.profiler import ProfilerActivity, profile
    for _ in range(5):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            fn()
            torch.cuda.synchronize()
        names = {k for k in KRYLOV for e in p.events() if k in e.name}
        if names:
            break
    return names


def _solve(shapes, kind, dtype, mode):
    """Solutions and reports of the systems of `shapes`, each with a right-hand side of its own (the same in every batch),
    the Krylov kernel that ran, and the FP64 residual over its bound (tolerance plus the drift of the recurrence)."""
    from pict_b200 import PISOtorch as P
    from pict_b200 import _lib
    from pict_b200.batch import BatchDomain
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    dom = BatchDomain([build_product(_box(s), dtype) for s in shapes], order="given")
    n, sims, D = dom.getTotalSize(), dom._sim_cells.cpu().numpy(), len(shapes[0])
    dt = 1e-3
    _lib.check(lib.pict_setup_advection(ctypes.byref(dom._desc), dt, st), "advection")
    _lib.check(lib.pict_copy_velocity_result_from_blocks(ctypes.byref(dom._desc), st), "copy")
    _lib.check(lib.pict_setup_pressure_correction(ctypes.byref(dom._desc), dt, 0, 0, st), "pressure")
    coef = (dom.P if kind == "cg" else dom.C).coef.clone().reshape(2 * D + 1, n)
    nrhs = 1 if kind == "cg" else D
    parts = []
    for s, s0, s1 in zip(shapes, sims[:-1], sims[1:]):
        g = torch.Generator().manual_seed(sum(s))
        b = torch.randn((nrhs, int(s1 - s0)), generator=g, dtype=torch.float64)
        b -= b.mean(dim=1, keepdim=True)                        # inside the range of the singular operator
        coef[:, s0:s1] /= coef[0, s0:s1].abs().max().clone()    # its own scale, alone and in the batch
        parts.append(b.to("cuda", dtype))
    b = torch.cat(parts, dim=1).contiguous()
    tol = 1e-4 if dtype == torch.float32 else 1e-9
    x = torch.zeros_like(b)
    prm = P._solve_params(nrhs, 5000, tol, 1, kind != "cg", False, x_zero=True, variant=1 if kind == "cg" else 0)
    infos = []

    def solve():
        x.zero_()
        infos[:] = P.decode_infos(P.solve_stencil(dom, coef.reshape(-1), b, x, prm))
    try:
        lib.pict_krylov_set_cluster_mode(mode)
        names = _kernels(solve)
    finally:
        lib.pict_krylov_set_cluster_mode(1)
    assert len(names) == 1, names
    assert all(i.converged and i.status == 0 for i in infos), infos
    A = _matrix(dom, coef, False)
    xd, bd = x.double().cpu().numpy(), b.double().cpu().numpy()
    eps = torch.finfo(dtype).eps
    drift = 200 * eps * abs(A).sum(axis=1).max() * np.abs(xd).max()
    for c in range(nrhs):
        r = bd[c] - A @ xd[c]
        for s0, s1 in zip(sims[:-1], sims[1:]):
            assert np.sqrt((r[s0:s1] ** 2).mean()) <= tol + drift
    out = [(x[:, s0:s1].clone(), [i.usedIterations for i in infos[k * nrhs:(k + 1) * nrhs]])
           for k, (s0, s1) in enumerate(zip(sims[:-1], sims[1:]))]
    return out, names.pop()


def _limit(kind, dims, dtype):
    """Cells of the largest system that is solved on chip (pict_krylov_set_cluster_mode)."""
    if kind == "cg":
        return 65536 if dtype == torch.float32 else 32768
    return 32768 if dims == 2 and dtype == torch.float32 else 16384


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("shape", [(64, 64), (128, 128), (129, 128), (256, 128), (257, 128), (256, 256), (257, 256),
                                   (25, 25, 26), (26, 25, 26), (32, 32, 32), (33, 32, 32), (40, 40, 41)], ids=str)
def test_kernel_that_runs(shape, kind, dtype):
    n = int(np.prod(shape))
    on_chip = n <= _limit(kind, len(shape), dtype)
    beyond = "k_cg1_cluster" if kind == "cg" else "k_bicgstab<"
    want = "k_cg1_resident" if kind == "cg" else "k_bicgstab_resident"
    assert _solve([shape], kind, dtype, 1)[1] == (want if on_chip else beyond)
    assert _solve([shape], kind, dtype, 0)[1] == ("k_cg1<" if kind == "cg" else "k_bicgstab<")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("mode,more", [(0, []), (0, [(40, 40), (300, 300)]), (1, []), (1, [(120, 120)])],
                         ids=["grid", "grid beside a large one", "on chip", "on chip beside a larger one"])
def test_members_equal_their_solo_solves(mode, more, kind, dtype):
    """Bit for bit, on the grid whatever else is in the batch, and among on-chip solves whatever form the largest member
    takes."""
    shapes = (SMALL + more) if mode == 0 else SMALL[:8 - len(more)] + more
    batch, name = _solve(shapes, kind, dtype, mode)
    if mode == 1:
        assert "resident" in name
    for s, (x, its) in zip(SMALL[:8 - len(more)], batch):
        (solo,), name1 = _solve([s], kind, dtype, mode)
        assert name1 == name and torch.equal(solo[0], x) and solo[1] == its, s


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("more", [[(40, 40)], [(300, 300)]], ids=["nine systems", "one too large"])
def test_members_beside_a_batch_that_is_solved_otherwise(more, kind, dtype):
    """With the default choice a ninth system, or one above the on-chip limit, sends the whole batch to another kernel: the
    same solutions to the tolerance (asserted in _solve for both), in as many iterations or one or two more or fewer (a
    stop at a residual of the same size, summed in another order)."""
    shapes = SMALL + more if more == [(40, 40)] else SMALL[:7] + more
    batch, name = _solve(shapes, kind, dtype, 1)
    assert "resident" not in name
    for s, (x, its) in zip(SMALL[:7], batch):
        (solo,), name1 = _solve([s], kind, dtype, 1)
        assert "resident" in name1
        assert all(abs(a - b) <= 2 for a, b in zip(its, solo[1])), (s, its, solo[1])
