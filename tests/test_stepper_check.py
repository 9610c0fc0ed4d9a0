"""PISOStepper.check names every solve of the step that failed (CPU, with made-up solver reports)."""
import types

import pytest
import torch


def _stepper(adv, refine):
    from pict_b200.engine import PISOStepper
    block = lambda *n: types.SimpleNamespace(velocity=torch.zeros((1, len(n)) + tuple(reversed(n))))
    member = lambda *blocks: types.SimpleNamespace(getBlocks=lambda: list(blocks))
    st = object.__new__(PISOStepper)
    st.domain = types.SimpleNamespace(order=[1, 0], domains=[member(block(32, 32)), member(block(96, 40), block(8, 40))])
    st.dims, st.adv_tol, st.p_tol, st.refine_tol, st.pressure_first_solve = 2, 5e-7, 1e-6, 5e-10, False
    st.infos = lambda: (adv, [[]])
    st.refine_infos = lambda: [[refine]]
    return st


def _info(residual=1e-12, iterations=3, converged=True, finite=True, status=0):
    from pict_b200.PISOtorch import LinearSolverResultInfo
    inf = LinearSolverResultInfo(residual, iterations, converged, finite)
    inf.status = status
    return inf


def test_good_reports_are_returned():
    adv = [_info() for _ in range(4)]
    assert _stepper(adv, [_info(), _info()]).check()[0] is adv


def test_every_failed_solve_is_named():
    from pict_b200.engine import LinsolveError
    adv = [_info(), _info(), _info(), _info(float("nan"), 7, False, False)]
    bad = [_info(1e-3, 0, False, True, 1), _info(7.5e-10, 16, False)]
    with pytest.raises(LinsolveError) as e:
        _stepper(adv, bad).check()
    text = str(e.value)
    assert text.startswith("advection solve reported non-finite residual for RHS 3")
    assert "3 failed" in text
    assert "advection, system 1 (member 0, 32x32), tolerance 5e-07, residual nan after 7 iterations, status 0" in text
    assert "pressure 0 refinement 0, system 0 (member 1, 96x40, 8x40), tolerance 5e-10, residual 0.001 after 0 iterations, status 1" in text
    assert "pressure 0 refinement 0, system 1 (member 0, 32x32), tolerance 5e-10, residual 7.5e-10 after 16 iterations, status 0" in text


def test_a_long_list_is_cut():
    from pict_b200.engine import LinsolveError
    with pytest.raises(LinsolveError, match="and 12 more"):
        st = _stepper([], [_info(1.0, 1, False)] * 20)
        st._system_name = lambda s: "system %d" % s
        st.check()
