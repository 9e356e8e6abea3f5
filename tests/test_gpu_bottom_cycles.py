"""The cluster kernel for the bottom of the pressure cycle against the launch
sequence it replaces, at the sizes where its form changes (one or two leaves
per thread, the three shapes of the coarsest CG), and the coarsest solves
themselves against the oracle.  The kernel does the same operations in the same
order: bit-identical."""
import numpy as np
import pytest

from oracle.oracle import OraclePoisson
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


def droplets(n, count):
    rng = np.random.default_rng(3)
    balls = [(tuple(rng.uniform(0.06, 0.94, 3)), 0.05) for _ in range(count)]
    return scenes.sdf_box_scene(n, None, balls, 3, 1.0)


# (leaves, DOF) of the level next to the coarsest and of the coarsest: 40 / 1,896 DOF; 57 / 3,360; 61 / 1,039;
# 82 / 974; 21 / 650; 120 leaves are the most that fit: 84^3 has 122 on level 1, so its bottom is a level further down
@pytest.mark.parametrize("scene", [lambda: scenes.plain_poisson_scene(64, 3), lambda: scenes.plain_poisson_scene(80, 3),
                                   lambda: droplets(128, 110), lambda: droplets(160, 60),
                                   lambda: scenes.plain_poisson_scene(84, 3)],
                         ids=["one leaf, 4 x 512", "one leaf, 4 x 1024", "two leaves, 4 x 512", "two leaves, 2 x 512",
                              "four levels"])
def test_pressure_bottom_identical(gpu, monkeypatch, scene):
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver
    sc = scene()
    out = []
    for on in ("0", "1"):
        monkeypatch.setenv("UAAMG_BOTTOM", on)
        lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
        rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
        s = PoissonSolver(lap)
        z, p = s.precondition(rhs), lap.getZeroVectorGrid()
        st = s.solveMultigridPCG(p, rhs)
        d = gpu.from_numpy(rhs).cuda()
        bottom = any("bottom" in k for k in s.profile_pcg(gpu.zeros_like(d), d))
        out.append((z, p, st, s.mIterationTaken, bottom))
    (z0, p0, st0, it0, b0), (z1, p1, st1, it1, b1) = out
    assert not b0 and b1
    assert np.array_equal(z0, z1) and np.array_equal(p0, p1) and (st0, it0) == (st1, it1) and st0 == 0


def test_pressure_coarsest_solve_of_each_shape(gpu):
    """776, 1,896 and 3,360 DOF: the three shapes, with the oracle's solve's tolerance (another summation order)."""
    from uaamg_b200.poisson import LaplacianWithLevel
    for n in (48, 64, 40):
        sc = scenes.plain_poisson_scene(n, 1)
        lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
        ref = OraclePoisson(sc.phi, sc.face_weights, sc.dt, sc.dx)
        lc = ref.num_levels - 1
        b = np.random.default_rng(60).uniform(-1, 1, ref.zeros(lc).shape).astype(np.float32)
        b[ref.dof_index(lc) < 0] = 0
        g, c = lap.coarsest_solve(b), ref.coarsest_solve(b)
        assert np.linalg.norm(g - c) <= 1e-4 * np.linalg.norm(c)
