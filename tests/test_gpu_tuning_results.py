"""No kernel-shape setting changes a result, on a level 0 large enough that its
dot products are summed by the marching kernels' blocks (8,192 leaves): solves
with every threshold out of reach, and with every threshold at its lowest, equal
the default ones bit for bit."""
import numpy as np
import pytest

from uaamg_b200 import autotune, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu tests need a CUDA device")
    from uaamg_b200 import build
    build.build()
    return torch


@pytest.fixture(scope="module")
def problem(gpu):
    from uaamg_b200.poisson import LaplacianWithLevel
    sc = scenes.large_poisson_scene(n=216, seed=2)
    lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
    assert lap.leaf_count(0) >= 8192
    return lap, lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)


FORMS = [{}, {"staged_min_leaves": autotune.NEVER, "split_min_leaves": autotune.NEVER, "pipe_min_leaves": autotune.NEVER},
         {"staged_min_leaves": 1, "split_min_leaves": 1, "pipe_min_leaves": 1}]


@pytest.mark.parametrize("smoother,precision", [(0, None), (1, None), (2, None), (3, None), (0, "fp16"), (0, "bf16")])
def test_settings_leave_results_alone(problem, smoother, precision):
    from uaamg_b200.poisson import PoissonSolver
    lap, rhs = problem
    start = autotune.get()
    got = []
    s = PoissonSolver(lap)
    s.mSmoother = PoissonSolver.SmootherOption(smoother)
    s.precondition(rhs)  # SPAI0's first cycle of a hierarchy builds its coefficients as it goes
    try:
        for form in FORMS:
            autotune.set({**start, **form})
            p = lap.getZeroVectorGrid()
            st = s.solveMultigridPCGMixed(p, rhs, precision) if precision else s.solveMultigridPCG(p, rhs)
            got.append((st, s.mIterationTaken, p))
    finally:
        autotune.set(start)
    for st, it, p in got[1:]:
        assert (st, it) == got[0][:2] and np.array_equal(p, got[0][2])
    assert precision or got[0][0] == 0  # (a 16-bit cycle is no fit preconditioner for every domain)
