"""Freed device blocks are kept and given to later allocations: results stay
the same when handles of several sizes are made and dropped in turn, on own
and caller's streams and from two threads, and what is kept stays bounded."""
import threading

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


def pressure(n, stream=None):
    from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver
    sc = scenes.plain_poisson_scene(n, n)
    lap = LaplacianWithLevel.createPressurePoissonLaplacianWithRhs(
        sc.phi, sc.face_weights, sc.vx, sc.vy, sc.vz, sc.solid_velocity, sc.dt, sc.dx, stream=stream)
    p = lap.getZeroVectorGrid()
    assert PoissonSolver(lap).solveMultigridPCGResident(p) == 0
    return p


def viscosity(n, stream=None):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.plain_viscosity_scene(n, n)
    lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx,
                                              stream=stream)
    rhs, x = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity), lv.gather_velocity(sc.u, sc.v, sc.w)
    simd_viscosity3d(lv).pcg_solve(x, 1e-6, rhs)
    return x


def test_handles_in_turn(gpu):
    jobs = [(pressure, 40), (viscosity, 16), (pressure, 48), (viscosity, 24), (pressure, 32)]
    want = [f(n) for f, n in jobs]
    side = gpu.cuda.Stream()
    for turn in range(3):
        stream = side.cuda_stream if turn == 1 else None  # a caller's stream, then own ones again
        for (f, n), w in zip(jobs, want):
            assert np.array_equal(f(n, stream), w)
    del side
    failed = []

    def work(order):
        for _ in range(3):
            for k in order:
                f, n = jobs[k]
                if not np.array_equal(f(n), want[k]):
                    failed.append(k)

    threads = [threading.Thread(target=work, args=(o,)) for o in ((0, 1, 2, 3, 4), (4, 3, 2, 1, 0))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    # many handles alive at once, then dropped: later ones still agree
    from uaamg_b200.poisson import LaplacianWithLevel
    sc = scenes.plain_poisson_scene(32, 32)
    kept = [LaplacianWithLevel.createPressurePoissonLaplacian(sc.phi, sc.face_weights, sc.dt, sc.dx) for _ in range(24)]
    assert np.array_equal(pressure(40), want[0])
    del kept
    assert np.array_equal(viscosity(24), want[3]) and np.array_equal(pressure(48), want[2])
