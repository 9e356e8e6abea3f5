"""A change of bottom_cycle applies to the next solve of a handle that exists
already, as every other kernel-shape setting does: the cluster launch appears
and disappears with it, in host-driven solves and in replayed graphs, and the
results stay equal bit for bit."""
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


@pytest.mark.parametrize("graph", [0, 2])
def test_bottom_cycle_follows_the_setting(gpu, graph):
    from uaamg_b200 import autotune
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver
    sc = scenes.plain_poisson_scene(n=64, seed=3)
    lap = LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx)
    rhs = lap.createPressurePoissonRightHandSide(sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt)
    s = PoissonSolver(lap)
    s.use_graph = graph
    start = autotune.get()
    d = gpu.from_numpy(rhs).cuda()
    label = f"L{lap.num_levels() - 2} bottom (2 visits + coarsest)"
    launches, want = {}, None
    try:
        for on in (1, 0, 1):
            autotune.set({"bottom_cycle": on})
            p = lap.getZeroVectorGrid()
            before = s.kernel_launches
            assert s.solveMultigridPCG(p, rhs) == 0
            n = s.kernel_launches - before
            assert launches.setdefault(on, n) == n
            want = p if want is None else want
            assert np.array_equal(p, want)
            assert (label in s.profile_pcg(gpu.zeros_like(d), d)) == bool(on)
    finally:
        autotune.set(start)
    assert launches[1] < launches[0]
