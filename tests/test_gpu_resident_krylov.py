"""Cluster-resident CG and BiCGStab (GPU) against the same recurrences on the persistent grid, at the sizes where
the split changes: systems smaller than the cluster, the last size of each cells-per-thread step, one cell more,
the largest resident system and the first that falls back; FP32 / FP64, plain and transposed, from zero and from a
guess, with connected, rotated and periodic faces and several uneven systems in one launch.

Both kernels stop at the same RMS residual and sum in different orders: iteration counts may differ by one (BiCGStab two)
or, in long solves, by 3%, and the residual of either solution, recomputed in FP64, is below the tolerance plus the drift of the recurrence (a few
hundred roundings of the solution's size times the largest row sum)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from setups import build_product, case, lid_cavity, tensor_grid

pytestmark = pytest.mark.gpu


def _box(shape):
    axes = [np.linspace(0, 1, s + 1) for s in shape]
    rng = np.random.default_rng(sum(shape))
    vel = rng.standard_normal((1, len(shape)) + tuple(reversed(shape))) * 0.1
    spec = dict(dims=len(shape), viscosity=1e-2, blocks=[dict(coords=tensor_grid(*axes), velocity=vel)],
                ops=[("close_all", 0)] + ([("periodic", 0, "x")] if shape[0] % 2 else []))
    return spec


def _domain(layout, dtype):
    if isinstance(layout, tuple):
        return build_product(_box(layout), dtype)
    if layout == "batch":
        from pict_b200.batch import BatchDomain
        doms = [build_product(lid_cavity(n, viscosity=1e-3), dtype) for n in (150, 91, 64, 17, 3)]
        return BatchDomain(doms)
    return build_product(case(layout), dtype)


def _matrix(dom, coef, transpose):
    K, n = coef.shape
    c, nb = coef.double().cpu().numpy(), dom._nbr.cpu().numpy()
    i = np.arange(n)
    rows, cols, vals = [i], [i], [c[0]]
    for f in range(K - 1):
        ok = nb[f] >= 0
        rows.append(i[ok])
        cols.append(nb[f][ok])
        vals.append(c[f + 1][ok])
    A = sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(n, n))
    return A.T.tocsr() if transpose else A


LAYOUTS = [(5, 3), (64, 128), (127, 65), (128, 128), (181, 91), (256, 128), (331, 100), (256, 256), (257, 256),
           (20, 20, 20), (25, 27, 31), (32, 32, 32), (33, 32, 32), "batch", "ring4_2d", "twoblock2d_rotated", "twoblock3d"]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("layout", LAYOUTS, ids=str)
def test_resident_solves_match_grid_solves(layout, dtype):
    from pict_b200 import PISOtorch as P
    from pict_b200 import _lib
    lib = _lib.load()
    dom = _domain(layout, dtype)
    D, n = dom.getSpatialDims(), dom.getTotalSize()
    st = torch.cuda.current_stream().cuda_stream
    # a time step at which the off-diagonal row sums of C are about half its diagonal: every iteration then at least
    # halves the residual, so a solve whose sums differ by roundings stops within one or two iterations of another
    h2 = sum(4.0 / (min(b.transform.reshape(-1, 2 * D * D + 1)[:, a * D + a].abs().min().item(), 1.0) ** 2
                    if b.transform is not None else 1.0) for b in dom.getBlocks()[:1] for a in range(D))
    dt = 0.5 / (1e-2 * h2 + np.sqrt(h2))
    _lib.check(lib.pict_setup_advection(ctypes.byref(dom._desc), dt, st), "advection")
    _lib.check(lib.pict_copy_velocity_result_from_blocks(ctypes.byref(dom._desc), st), "copy")
    _lib.check(lib.pict_setup_pressure_correction(ctypes.byref(dom._desc), dt, 0, 0, st), "pressure")
    g = torch.Generator().manual_seed(1)
    sims = dom._sim_cells.cpu().numpy()
    for kind in ("cg", "bicgstab"):
        nrhs = 1 if kind == "cg" else D
        coef = (dom.P if kind == "cg" else dom.C).coef.clone()
        b = torch.randn((nrhs, n), generator=g, dtype=torch.float64)
        if kind == "cg":  # inside the range of the singular operator
            for s0, s1 in zip(sims[:-1], sims[1:]):
                b[:, s0:s1] -= b[:, s0:s1].mean()
        b = (b * float(coef[0].abs().max())).to("cuda", dtype).contiguous()
        scale = float(b.double().norm()) / np.sqrt(b.numel())
        tol = (1e-4 if dtype == torch.float32 else 1e-10) * scale
        guess = torch.randn((nrhs, n), generator=g, dtype=torch.float64).to("cuda", dtype)
        for transpose in (False, True):
            A = _matrix(dom, coef.reshape(2 * D + 1, n), transpose)
            for zero in (True, False):
                out = []
                for mode in (0, 2):
                    x = torch.zeros_like(b) if zero else guess.clone()
                    prm = P._solve_params(nrhs, 5000, tol, 1, kind != "cg", transpose, x_zero=zero,
                                          variant=1 if kind == "cg" else 0)
                    try:
                        lib.pict_krylov_set_cluster_mode(mode)
                        infos = P.decode_infos(P.solve_stencil(dom, coef, b, x, prm))
                    finally:
                        lib.pict_krylov_set_cluster_mode(1)
                    assert all(i.converged and i.isFiniteResidual and i.status == 0 for i in infos), (kind, mode, infos)
                    out.append((x.double().cpu().numpy(), [i.usedIterations for i in infos]))
                (xg, ig), (xr, ir) = out
                slack = 1 if kind == "cg" else 2
                assert all(abs(p - q) <= max(slack, 0.03 * p) for p, q in zip(ig, ir)), (kind, transpose, zero, ig, ir)
                eps = np.finfo(np.float32 if dtype == torch.float32 else np.float64).eps
                for x in (xg, xr):
                    drift = 200 * eps * abs(A).sum(axis=1).max() * np.abs(x).max()
                    for c in range(nrhs):
                        r = b[c].double().cpu().numpy() - A @ x[c]
                        for s0, s1 in zip(sims[:-1], sims[1:]):
                            assert np.sqrt((r[s0:s1] ** 2).mean()) <= tol + drift, (kind, transpose, zero)


def _small(kind, dtype):
    """Matrix and right-hand side of a batch of three boxes, on-chip at every form of the kernels."""
    from pict_b200 import _lib
    from pict_b200.batch import BatchDomain
    lib = _lib.load()
    dom = BatchDomain([build_product(_box(s), dtype) for s in ((120, 100), (33, 40), (9, 7))])
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.pict_setup_advection(ctypes.byref(dom._desc), 1e-3, st), "advection")
    _lib.check(lib.pict_copy_velocity_result_from_blocks(ctypes.byref(dom._desc), st), "copy")
    _lib.check(lib.pict_setup_pressure_correction(ctypes.byref(dom._desc), 1e-3, 0, 0, st), "pressure")
    coef = (dom.P if kind == "cg" else dom.C).coef.clone()
    coef /= coef[:dom.getTotalSize()].abs().max()
    g = torch.Generator().manual_seed(4)
    b = torch.randn((1 if kind == "cg" else 2, dom.getTotalSize()), generator=g, dtype=torch.float64)
    sims = dom._sim_cells.cpu().numpy()
    for s0, s1 in zip(sims[:-1], sims[1:]):
        b[:, s0:s1] -= b[:, s0:s1].mean(dim=1, keepdim=True)
    return dom, coef, b.to("cuda", dtype).contiguous()


def _both(dom, coef, b, x0, kind, maxit, tol):
    """Reports and solutions on the grid and on chip."""
    from pict_b200 import PISOtorch as P
    from pict_b200 import _lib
    lib = _lib.load()
    out = []
    for mode in (0, 2):
        x = x0.clone()
        prm = P._solve_params(b.shape[0], maxit, tol, 1, kind != "cg", False, x_zero=False, variant=1 if kind == "cg" else 0)
        try:
            lib.pict_krylov_set_cluster_mode(mode)
            infos = P.decode_infos(P.solve_stencil(dom, coef, b, x, prm))
        finally:
            lib.pict_krylov_set_cluster_mode(1)
        out.append(([(i.usedIterations, i.converged, i.isFiniteResidual, i.status) for i in infos], x))
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
def test_reports_at_the_edges(kind, dtype):
    """A right-hand side of zeros (in one system only), a cap on the iterations, no iterations at all, and a start that
    already solves the system: the reports of the grid kernels, and their solutions."""
    dom, coef, b = _small(kind, dtype)
    s1 = int(dom._sim_cells[1])
    g = torch.Generator().manual_seed(6)
    x0 = torch.randn(b.shape, generator=g, dtype=torch.float64).to("cuda", dtype)
    # 200 roundings of the largest value for runs of the same few iterations
    close = lambda u, v: float((u - v).abs().max()) <= 200 * torch.finfo(dtype).eps * float(v.abs().max())
    tol = 1e-4 if dtype == torch.float32 else 1e-9
    zero = b.clone()
    zero[:, :s1] = 0.0
    (ig, xg), (ir, xr) = _both(dom, coef, zero, x0, kind, 3, 1e-30)
    assert ig == ir and close(xr, xg) and float(xr[:, :s1].abs().max()) == 0.0
    (ig, xg), (ir, xr) = _both(dom, coef, b, x0, kind, 5, 1e-30)
    assert ig == ir and not any(c for _, c, _, _ in ir) and close(xr, xg)
    (ig, xg), (ir, xr) = _both(dom, coef, b, x0, kind, 0, tol)
    assert ig == ir and torch.equal(xg, x0) and torch.equal(xr, x0)
    (ig, xg), _ = _both(dom, coef, b, x0, kind, 5000, tol)
    assert all(c for _, c, _, _ in ig)
    (ig, x1), (ir, x2) = _both(dom, coef, b, xg, kind, 5000, 10 * tol)
    assert ig == ir and all(c for _, c, _, _ in ir) and close(x2, x1)
