"""The multigrid PCG with its kernels launched dependently (each starts before its predecessor has ended) and one after
the other (GPU): the same kernels on the same operands, so fields and reports are equal bit for bit, step by step, over
batches of uneven cavities whose systems converge at different iterations."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(seed, dependent, graph):
    import bench
    from pict_b200 import _lib
    from pict_b200.batch import BatchDomain
    from pict_b200.engine import PISOStepper
    lib = _lib.load()
    rng = np.random.default_rng(seed)
    sides = np.rint(np.exp(rng.uniform(np.log(32), np.log(256), 40))).astype(int)
    nu = np.exp(-rng.uniform(np.log(100), np.log(5000), 40))
    try:
        lib.pict_mg_set_dependent_launch(dependent)
        b = BatchDomain([bench.make_cavity_domain(int(n), float(v), torch.float32) for n, v in zip(sides, nu)],
                        time_steps=[0.5 / n for n in sides])
        st = PISOStepper(b, time_step=0.01, advection_tol=5e-7, pressure_tol=1e-6, pressure_refine=1, refine_tol=5e-10,
                         warm_start_pressure="increment", refine_solver="auto", mg_iterations=16,
                         pressure_first_solve=False, warm_start_advection="increment")
        assert st._mg is not None
        out = []
        if graph:
            st.capture(steps=1)
        for _ in range(6):
            st.replay() if graph else st.step()
            st.check()
            out.append([(i.usedIterations, i.finalResidual) for row in st.refine_infos() for r in row for i in r])
        return out, [t.clone() for d in b.getBlocks() for t in (d.velocity, d.pressure)]
    finally:
        lib.pict_mg_set_dependent_launch(1)


@pytest.mark.parametrize("graph", [False, True], ids=["launched", "captured"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_dependent_launches_equal_plain_ones(seed, graph):
    reports, fields = _run(seed, 1, graph)
    plain, plain_fields = _run(seed, 0, graph)
    assert reports == plain
    assert all(torch.equal(a, b) for a, b in zip(fields, plain_fields))
