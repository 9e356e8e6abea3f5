"""The cluster kernels for the bottom of the cycles against the launch
sequences they replace, at the sizes where their forms change: pressure
(k_bottom: one or two leaves per thread, the three shapes of the coarsest CG)
and viscosity (k_vbottom: level next to the coarsest as the top level or below
it, the coarsest CG in one CTA or over eight, a level that does not fit), and
the coarsest solves themselves against the oracle.  The kernels do the same
operations in the same order: bit-identical."""
import numpy as np
import pytest

from oracle.oracle import OraclePoisson, OracleViscosity
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


# coarsest DOF: 884 under a top level of 5,668; 2,836 under 19,208; 880 under 5,836; 1,668 under 11,568; 2,520 under
# 19,028; 3,852 under 29,948, which does not fit
@pytest.mark.parametrize("n,fits", [(16, True), (24, True), (32, True), (40, True), (48, True), (56, False)])
def test_viscosity_bottom_identical(gpu, monkeypatch, n, fits):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.plain_viscosity_scene(n=n, seed=2)
    out = []
    for on in ("0", "1"):
        monkeypatch.setenv("UAAMG_VISC_BOTTOM", on)
        lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
        rhs = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)
        s = simd_viscosity3d(lv)
        z = s.precondition(rhs)
        x = lv.gather_velocity(sc.u, sc.v, sc.w)
        st = s.pcg_solve(x, 1e-6, rhs)
        d, d0 = gpu.from_numpy(rhs).cuda(), gpu.zeros(rhs.shape, device="cuda")
        bottom = any("bottom" in k for k in s.profile_pcg(d0, d, 1e-6))
        out.append((z, x, st, s.m_iteration, bottom))
    (z0, x0, st0, it0, b0), (z1, x1, st1, it1, b1) = out
    assert not b0 and b1 == fits
    assert np.array_equal(z0, z1) and np.array_equal(x0, x1) and (st0, it0) == (st1, it1)


@pytest.mark.parametrize("n", [24, 32, 56])
def test_viscosity_coarsest_solve_bit_exact(gpu, n):
    from uaamg_b200.viscosity import L_with_level
    sc = scenes.plain_viscosity_scene(n=n, seed=2)
    lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
    ref = OracleViscosity(sc.liquid_phi, sc.solid_phi, sc.viscosity, sc.dt, sc.rho, sc.dx)
    lc = lv.num_levels() - 1
    b = np.random.default_rng(61).uniform(-1, 1, ref.zeros(lc).shape).astype(np.float32)
    b[ref.dof_index(lc) < 0] = 0
    for rhs in (b, np.zeros_like(b)):
        assert np.array_equal(lv.solve_exact(rhs), ref.coarsest_solve(rhs))
