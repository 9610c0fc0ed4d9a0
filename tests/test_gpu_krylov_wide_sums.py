"""Inner products of the persistent Krylov kernels on either side of the tile count above which a whole CTA sums a
system's partials (GPU): 512 and 513 tiles, which is also one step of the CTA's threads and one more, 546, half as many,
and one tile, several of them in one CTA's slots.  A system's sums do not depend on the others of a batch, so a batched solve equals the solo solve bit for
bit; the residual, recomputed in FP64, is below the tolerance plus the drift of the recurrence (a few hundred roundings
of the solution's size times the largest row sum)."""
import ctypes

import numpy as np
import pytest
import torch

from setups import build_product
from test_gpu_resident_krylov import _box, _matrix

pytestmark = pytest.mark.gpu

TILE = 32
SHAPES = [(192, 91), (513, 32), (128, 128), (91, 91), (257, 32), (128, 64), (6, 5)]   # 546, 513, 512, 259, 257, 256, 1 tiles


def _solve(shapes, rhs, tol, kind, variant, dtype):
    """The systems of `shapes` in one launch on the persistent grid: the solution of each (and the tolerance)."""
    from pict_b200 import PISOtorch as P
    from pict_b200 import _lib
    from pict_b200.batch import BatchDomain
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    nrhs = 1 if kind == "cg" else 2
    dom = BatchDomain([build_product(_box(s), dtype) for s in shapes], order="given")
    dom.set_tile_cells(TILE)
    n, sims = dom.getTotalSize(), dom._sim_cells.cpu().numpy()
    dt = 1e-3
    _lib.check(lib.pict_setup_advection(ctypes.byref(dom._desc), dt, st), "advection")
    _lib.check(lib.pict_copy_velocity_result_from_blocks(ctypes.byref(dom._desc), st), "copy")
    _lib.check(lib.pict_setup_pressure_correction(ctypes.byref(dom._desc), dt, 0, 0, st), "pressure")
    coef = (dom.P if kind == "cg" else dom.C).coef.clone()
    diag = coef.reshape(5, n)[0]
    # each system's right-hand side scaled by its own diagonal, so that it is the same alone and in the batch
    b = torch.cat([rhs[s] * diag[s0:s1].abs().max() for s, s0, s1 in zip(shapes, sims[:-1], sims[1:])], dim=1).contiguous()
    if tol is None:
        tol = (1e-4 if dtype == torch.float32 else 1e-9) * float(diag.abs().max())
    x = torch.zeros_like(b)
    prm = P._solve_params(nrhs, 3000, tol, 1, kind != "cg", False, x_zero=True, variant=variant if kind == "cg" else 0)
    try:
        lib.pict_krylov_set_cluster_mode(0)
        lib.pict_krylov_set_bicgstab_variant(variant if kind != "cg" else 0)
        infos = P.decode_infos(P.solve_stencil(dom, coef, b, x, prm))
    finally:
        lib.pict_krylov_set_cluster_mode(1)
        lib.pict_krylov_set_bicgstab_variant(0)
    assert all(i.converged and i.isFiniteResidual for i in infos), infos
    A = _matrix(dom, coef.reshape(5, n), False)
    for c in range(nrhs):
        xc = x[c].double().cpu().numpy()
        r = b[c].double().cpu().numpy() - A @ xc
        drift = 200 * torch.finfo(dtype).eps * abs(A).sum(axis=1).max() * np.abs(xc).max()
        for s0, s1 in zip(sims[:-1], sims[1:]):
            assert np.sqrt((r[s0:s1] ** 2).mean()) <= tol + drift
    return [x[:, s0:s1] for s0, s1 in zip(sims[:-1], sims[1:])], tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind,variant", [("cg", 0), ("cg", 1), ("bicgstab", 0), ("bicgstab", 1), ("bicgstab", 2)])
def test_wide_systems_batched_equal_solo(kind, variant, dtype):
    g = torch.Generator().manual_seed(3)
    rhs = {}
    for s in SHAPES:
        b = torch.randn((1 if kind == "cg" else 2, s[0] * s[1]), generator=g, dtype=torch.float64)
        rhs[s] = (b - b.mean(dim=1, keepdim=True)).to("cuda", dtype)   # inside the range of the singular operator
    xs, tol = _solve(SHAPES, rhs, None, kind, variant, dtype)
    for s, xb in zip(SHAPES, xs):
        (xa,), _ = _solve([s], rhs, tol, kind, variant, dtype)
        assert torch.equal(xa, xb), s
