"""Viscosity passes that take plain leaves apart, against the general passes.

A level's leaves are plain (all DOF, constant coefficients) or general; from a
size on, a pass handles the two kinds differently in one launch.  Every value is
computed by the same operations in the same order, so the preconditioner and a
whole solve are equal bit for bit.  Sizes: one with hardly a plain leaf, an odd
one, and one with plain leaves on two levels; the number of lanes without work
differs in each.
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


@pytest.mark.parametrize("n,fill", [(24, 0.4), (53, 0.9), (96, 0.8)])
def test_plain_leaves_equal(gpu, monkeypatch, n, fill):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.viscosity_box_scene(n, fill, [((0.5, 0.7, 0.5), 0.15)], 2, 1e3)
    monkeypatch.setenv("UAAMG_VISC_FUSED_RB_LEAVES", "0")
    out = []
    for leaves in ("1", str(2**31 - 1)):
        monkeypatch.setenv("UAAMG_VISC_PLAIN_LEAVES", leaves)
        lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
        rhs = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)
        x = lv.gather_velocity(sc.u, sc.v, sc.w)
        s = simd_viscosity3d(lv)
        z = s.precondition(rhs)
        st = s.pcg_solve(x, 1e-6, rhs)
        out.append((z, x, st, s.m_iteration))
    (z0, x0, *a), (z1, x1, *b) = out
    assert np.array_equal(z0, z1)
    assert a == b and a[0] == 0
    assert np.array_equal(x0, x1)


def test_precondition_zero_outside_dof(gpu):
    """Level 0 is the bottom level at 24^3: the cycle writes its DOF only, and the
    result is zero elsewhere whatever the memory held before."""
    import gc
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.plain_viscosity_scene(n=24, seed=2)
    for _ in range(3):
        lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
        assert lv.num_levels() == 2
        rhs = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)
        s = simd_viscosity3d(lv)
        z = s.precondition(np.ones_like(rhs))
        assert not z[np.asarray(lv.dof_index(0)).reshape(z.shape) < 0].any()
        x = lv.gather_velocity(sc.u, sc.v, sc.w)
        s.pcg_solve(x, 1e-6, rhs)
        del s, lv
        gc.collect()
