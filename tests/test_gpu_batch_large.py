"""Batches that hold instances of at least 8,192 level-0 leaves.

A standalone solve adds such a level's dot products by the marching kernels'
blocks (two planes of a leaf per half-warp, from 24,576 leaves on whole leaves),
the batch leaf by leaf.  The sums are FP64 and their scalars FP32, so on these
inputs every instance's result, iterations and status are still its standalone
solve's, bit for bit, whatever the others are.
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
    out = [scenes.plain_poisson_scene(n=40, seed=1), scenes.large_poisson_scene(n=300, seed=2),
           scenes.sdf_box_scene(12, None, [((0.5, 0.5, 0.5), 0.3)], 11),  # one-level hierarchy
           scenes.large_poisson_scene(n=211, seed=3), scenes.plain_poisson_scene(n=107, seed=5)]
    return out


@pytest.mark.parametrize("members", [(0, 1, 2, 3, 4), (3,), (1, 3)])
@pytest.mark.parametrize("smoother", [0, 1, 2, 3])
def test_large_instances_equal_standalone(mix, smoother, members):
    from uaamg_b200.batch import PoissonBatch
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver

    def make(sc):
        lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
        s = PoissonSolver(lap)
        s.mSmoother = PoissonSolver.SmootherOption(smoother)
        rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
        s.precondition(rhs)  # SPAI0's first cycle of a hierarchy builds its coefficients as it goes
        return lap, s, rhs

    made = [make(mix[i]) for i in members]
    nl = dict(zip(members, (m[0].leaf_count(0) for m in made)))
    assert 8192 <= nl[3] < 24576 and nl.get(1, 24576) >= 24576
    alone = []
    for lap, s, rhs in [make(mix[i]) for i in members]:
        p = lap.getZeroVectorGrid()
        alone.append((p, s.solveMultigridPCG(p, rhs), s.mIterationTaken))
    b = PoissonBatch([m[1] for m in made])
    b.mSmoother = made[0][1].mSmoother
    for turn in range(2):  # host-driven, then as a graph
        ps = [m[0].getZeroVectorGrid() for m in made]
        b.solveMultigridPCG(ps, [m[2] for m in made])
        for i, (p, st, it) in enumerate(alone):
            assert (b.status[i], b.mIterationTaken[i]) == (st, it), (i, turn)
            assert np.array_equal(ps[i], p), (i, turn)
