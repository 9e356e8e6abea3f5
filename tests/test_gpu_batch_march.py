"""Batches whose depths hold enough leaves for the marching sweeps.

From 1,024 leaves over all instances on, a depth's sweeps and restriction march
and its computed sources are stored first; coarsest systems of different size
classes share a launch.  Every instance's result, iterations and status are
still its standalone solve's, bit for bit.  The mix holds level counts from one
up, instances that stop early, and totals that leave the last warps idle.
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


@pytest.fixture(scope="module")
def mix(gpu):
    out = [scenes.plain_poisson_scene(n=n, seed=n) for n in (104, 107, 110, 113, 120, 128, 43, 64)]
    out.append(scenes.sdf_box_scene(12, None, [((0.5, 0.5, 0.5), 0.3)], 11))
    out.append(scenes.random_balls_scene(3, sides=(48,)))
    return out


@pytest.mark.parametrize("smoother", [0, 1, 2, 3])
def test_marching_batch_equals_standalone(mix, smoother):
    from uaamg_b200.batch import PoissonBatch
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver

    def make(sc):
        lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
        s = PoissonSolver(lap)
        s.mSmoother = PoissonSolver.SmootherOption(smoother)
        return lap, s, lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)

    alone, made = [], [make(sc) for sc in mix]
    assert sum(m[0].leaf_count(1) for m in made if m[0].num_levels() > 2) >= 1024
    for lap, s, rhs in [make(sc) for sc in mix]:
        p = lap.getZeroVectorGrid()
        alone.append((p, s.solveMultigridPCG(p, rhs), s.mIterationTaken))
    b = PoissonBatch([m[1] for m in made])
    b.mSmoother = made[0][1].mSmoother
    ps = [m[0].getZeroVectorGrid() for m in made]
    b.solveMultigridPCG(ps, [m[2] for m in made])
    for i, (p, st, it) in enumerate(alone):
        assert np.array_equal(ps[i], p), i
        assert (b.status[i], b.mIterationTaken[i]) == (st, it), i
