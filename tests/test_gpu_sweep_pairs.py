"""Two sweeps in one launch against a launch per sweep.

Levels of up to about 296 leaves run Jacobi sweeps, and the two colours of a
red-black sweep, in pairs.  A batch of one instance runs a launch per sweep with
the same operations, so the solves are equal bit for bit.  Level sizes: 5, 19 (24^3),
57, 13 (40^3), 284, 40, 8 (64^3), and 776 to 5 leaves (96^3, level 0 above the
pairs' range).
"""
import numpy as np
import pytest

from uaamg_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu tests need a CUDA device")
    from uaamg_b200 import build
    build.build()
    return torch


@pytest.mark.parametrize("smoother", [0, 1, 2])
@pytest.mark.parametrize("n", [24, 40, 64, 96])
def test_pairs_equal(gpu, n, smoother):
    from uaamg_b200.batch import PoissonBatch
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver
    sc = scenes.plain_poisson_scene(n=n, seed=n)
    got = []
    for batched in (False, True):
        lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
        rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
        s = PoissonSolver(lap)
        s.mSmoother = PoissonSolver.SmootherOption(smoother)
        p = lap.getZeroVectorGrid()
        if batched:
            b = PoissonBatch([s])
            b.mSmoother = s.mSmoother
            b.solveMultigridPCG([p], [rhs])
            got.append((p, b.status[0], b.mIterationTaken[0]))
        else:
            got.append((p, s.solveMultigridPCG(p, rhs), s.mIterationTaken))
    assert got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0])
