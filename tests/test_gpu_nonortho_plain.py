"""The direct form of the non-orthogonal terms for cells away from walls and connections (GPU) against the oracle's
corner walk, on grids whose axes are just long enough to hold such cells (3 cells between walls), periodic along
some or all axes, FP64, every flag that selects a term."""
import numpy as np
import pytest
import torch

import piso_oracle as po
from setups import build_oracle, build_product, tensor_grid

pytestmark = pytest.mark.gpu


def _spec(shape, periodic):
    rng = np.random.default_rng(sum(shape))
    D = len(shape)
    c = tensor_grid(*[np.linspace(0, 1, s + 1) for s in shape])
    old = c[0].copy()
    for a in range(D):
        c[0, a] += 0.1 * old[(a + 1) % D] + 0.03 * np.sin(2 * np.pi * old[(a + 1) % D])
    zyx = tuple(reversed(shape))
    visc = 1e-2 + 1e-2 * rng.random((1, 1) + zyx)
    ops = [("close_all", 0)] + [("periodic", 0, "xyz"[a]) for a in periodic]
    return dict(dims=D, viscosity=1e-2, ops=ops,
                blocks=[dict(coords=c, velocity=rng.standard_normal((1, D) + zyx), viscosity=visc,
                             pressure=rng.standard_normal((1, 1) + zyx))])


@pytest.mark.parametrize("flags", [25, 27, 19, 16, 8, 2, 1])
@pytest.mark.parametrize("shape,periodic", [((3, 3), ()), ((3, 4), (0,)), ((4, 3), (1,)), ((3, 3), (0, 1)), ((5, 3), (0, 1)),
                                            ((3, 3, 3), ()), ((4, 3, 3), (2,)), ((3, 3, 3), (0, 1, 2)), ((5, 3, 4), (0, 2))],
                         ids=str)
def test_plain_cells_match_the_corner_walk(shape, periodic, flags):
    from pict_b200 import PISOtorch as P
    spec = _spec(shape, periodic)
    D = len(shape)
    od, pd = build_oracle(spec), build_product(spec, torch.float64)
    pd.getBlock(0).pressure.copy_(torch.tensor(spec["blocks"][0]["pressure"], device="cuda"))
    ts = torch.tensor([0.01], dtype=torch.float64)
    P.SetupAdvectionMatrix(pd, ts, flags)
    P.CopyVelocityResultFromBlocks(pd)
    P.SetupAdvectionVelocity(pd, ts, flags)
    P.CopyPressureResultFromBlocks(pd)
    P.SetupPressureMatrix(pd, ts, flags)
    P.SetupPressureRHS(pd, ts, flags)
    C, A = po.advection_matrix(od, 0.01, flags)
    u = od.velocity_global()
    h = po.pressure_rhs(od, 0.01, C, A, u)
    div = po.pressure_rhs_nonortho(od, flags, po.divergence(od, h), A, spec["blocks"][0]["pressure"].reshape(-1))
    for name, got, ref in [("C", pd.C.coef, C), ("A", pd.A, A), ("rhs", pd.velocityRHS, po.advection_rhs(od, 0.01, flags, u)),
                           ("P", pd.P.coef, po.pressure_matrix(od, A, flags)), ("h", pd.pressureRHS, h),
                           ("div", pd.pressureRHSdiv, div)]:
        got = got.double().cpu().numpy().reshape(ref.shape)
        # a few dozen FP64 roundings of the largest entry
        assert np.abs(got - ref).max() <= 1e-14 * 30 * np.abs(ref).max(), (name, np.abs(got - ref).max())
