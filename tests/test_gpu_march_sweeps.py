"""The marching sweeps against the kernels with one block per leaf.

Which kernel sweeps a level is set by its size; ``uaamg_set_tuning`` moves the
line, so both forms run on the same hierarchy.  They do the same operations in
the same order, so every result here is equal bit for bit.  The domains take
levels from one leaf up, partly filled leaves at the surface and the walls,
plain leaves (all DOF, default coefficients) inside, level sizes that leave a
launch's last warps without work, and (344^3) a level whose half-warps march
through whole leaves instead of two planes.
"""
import numpy as np
import pytest

from uaamg_b200 import scenes

pytestmark = pytest.mark.gpu

NEVER = 1 << 30
MARCH = {"staged_min_leaves": 1, "pipe_min_leaves": 1, "bottom_cycle": 0}
LEAF = {"staged_min_leaves": NEVER, "pipe_min_leaves": NEVER, "bottom_cycle": 0}


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu tests need a CUDA device")
    from uaamg_b200 import build
    build.build()
    return torch


@pytest.fixture
def tuned(gpu):
    from uaamg_b200 import autotune
    start = autotune.get()
    yield autotune.set
    autotune.set(start)


def laplacian(sc):
    from uaamg_b200.poisson import LaplacianWithLevel
    return LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)


def rand_vec(lap, level, seed):
    act = np.asarray(lap.dof_index(level)) >= 0
    return (np.random.default_rng(seed).standard_normal(act.shape) * act).astype(np.float32)


@pytest.mark.parametrize("n,fill", [(24, 0.45), (43, 0.45), (90, 0.45), (344, 0.9)])
def test_sweeps_and_cycle_equal(tuned, n, fill):
    from uaamg_b200.poisson import PoissonSolver
    spheres = [((0.3, 0.6, 0.4), 0.2), ((0.7, 0.5, 0.6), 0.15)]
    lap = laplacian(scenes.sdf_box_scene(n, fill, spheres, 3, 1.0, name="boxes"))
    if n > 300:
        assert lap.leaf_count(0) >= 65536
    for l in range(lap.num_levels() if n < 300 else 1):
        x, b = rand_vec(lap, l, 10 + l), rand_vec(lap, l, 30 + l)
        for mode in ("jacobi", "residual", "laplacian", "red_gs", "black_gs"):
            got = []
            for form in (MARCH, LEAF):
                tuned(form)
                got.append(lap.apply(l, mode, x, b, weight=0.8571, w_sor=1.2))
            assert np.array_equal(*got), (l, mode)
    r = rand_vec(lap, 0, 50)
    for smoother in PoissonSolver.SmootherOption:
        s = PoissonSolver(lap)
        s.mSmoother = smoother
        s.precondition(r)  # SPAI0's first cycle of a hierarchy builds its coefficients as it goes
        got = []
        for form in (MARCH, LEAF):
            tuned(form)
            got.append(s.precondition(r))
        assert np.array_equal(*got), smoother


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("n", [104, 131])
def test_mixed_solve_equal(tuned, n, precision):
    """Levels of 1,024 to 8,191 leaves: the dot products keep their kernels, so
    the whole solve is equal, its status and iterations included."""
    from uaamg_b200.poisson import PoissonSolver
    sc = scenes.large_poisson_scene(n=n, seed=4)
    lap = laplacian(sc)
    assert 1024 <= lap.leaf_count(0) < 8192
    rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
    s = PoissonSolver(lap)
    got = []
    for staged in (64, NEVER):
        tuned({"staged_min_leaves": staged})
        p = lap.getZeroVectorGrid()
        status = s.solveMultigridPCGMixed(p, rhs, precision)  # (BF16 stagnates at 104^3 in both forms)
        got.append((p, status, s.mIterationTaken))
    assert got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("smoother", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [104, 131])
def test_solve_equal(tuned, n, smoother):
    """Level 0 of 1,024 to 8,191 leaves: the passes with dot products march too,
    with the one-leaf kernels' sums, so a whole solve is equal."""
    from uaamg_b200.poisson import PoissonSolver
    sc = scenes.large_poisson_scene(n=n, seed=4)
    got = []
    for staged in (64, NEVER):
        tuned({"staged_min_leaves": staged})
        lap = laplacian(sc)
        assert 1024 <= lap.leaf_count(0) < 8192
        rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
        s = PoissonSolver(lap)
        s.mSmoother = PoissonSolver.SmootherOption(smoother)
        p = lap.getZeroVectorGrid()
        got.append((p, s.solveMultigridPCG(p, rhs), s.mIterationTaken))
    assert got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0])
