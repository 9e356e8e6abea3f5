"""The FP64 coarsest solve of the 16-bit form at sizes around its launch shape.

Sixteen rows per block, 256 values of a row at a time: coarsest systems below
and above a block, with row and value remainders.  The 16-bit solve must stay
within the form's bounds of the FP32 solve (at most two iterations more, solution
within 1e-5), which a wrong coarsest solution would break.
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


@pytest.mark.parametrize("n", [23, 26, 33, 40, 47])
def test_coarsest_sizes(gpu, n):
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver
    sc = scenes.plain_poisson_scene(n=n, seed=n)
    lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
    assert lap.num_levels() >= 2
    rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
    s = PoissonSolver(lap)
    p32, pm = lap.getZeroVectorGrid(), lap.getZeroVectorGrid()
    assert s.solveMultigridPCG(p32, rhs) == 0
    it32 = s.mIterationTaken
    assert s.solveMultigridPCGMixed(pm, rhs, "fp16") == 0
    # (the direct solve may need fewer: FP32's ten coarsest CG steps leave 3,360 DOF unsolved at 40^3)
    assert s.mIterationTaken <= it32 + 2
    assert np.linalg.norm(pm - p32) <= 1e-5 * np.linalg.norm(p32)
