"""k_vbottom on a level whose groups of rows are very unequal: plates of liquid
a voxel apart from one another hold no faces, or a few doors' faces, of the
channel across them.  Passes over groups too small for every CTA of the cluster
follow one another; with the coarsest CG in one CTA (28^3) and over eight
(36^3).  The preconditioner and a whole solve equal the launch sequence's."""
import numpy as np
import pytest

from uaamg_b200 import scenes
from uaamg_b200.grids import dense_to_leaves

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu tests need a CUDA device")
    from uaamg_b200 import build
    build.build()
    return torch


def plates(n, doors):
    sc = scenes.viscosity_box_scene(n, 2.0, [], 2, 1e3)
    d = np.full((n + 16,) * 3, -3.0, np.float32)
    d[8:8 + n, 8:8 + n, 8:8 + n] = -0.5
    d[9:8 + n:2, 8:8 + n, 8:8 + n] = 0.1
    for k in range(doors):
        d[10 + 2 * k, 12 + 2 * k, 10 + k] = 0.1
    sc.solid_phi = dense_to_leaves((d * sc.dx).astype(np.float32), origin=(-8, -8, -8), background=-3.0 * sc.dx)
    return sc


@pytest.mark.parametrize("n,doors", [(28, 0), (28, 3), (36, 0), (36, 3)])
def test_uneven_groups_identical(gpu, monkeypatch, n, doors):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = plates(n, doors)
    out = []
    for on in ("0", "1"):
        monkeypatch.setenv("UAAMG_VISC_BOTTOM", on)
        lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
        bottom = lv.num_levels() - 2
        idx = np.asarray(lv.dof_index(bottom)).reshape(3, -1) >= 0
        assert idx[0].sum() <= 2 * doors and min(idx[1].sum(), idx[2].sum()) > 2000
        rhs = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)
        s = simd_viscosity3d(lv)
        z = s.precondition(rhs)
        x = lv.gather_velocity(sc.u, sc.v, sc.w)
        st = s.pcg_solve(x, 1e-6, rhs)
        d, d0 = gpu.from_numpy(rhs).cuda(), gpu.zeros(rhs.shape, device="cuda")
        ran = any("bottom" in k for k in s.profile_pcg(d0, d, 1e-6))
        out.append((z, x, st, s.m_iteration, ran))
    (z0, x0, st0, it0, r0), (z1, x1, st1, it1, r1) = out
    assert not r0 and r1
    assert np.array_equal(z0, z1) and np.array_equal(x0, x1) and (st0, it0) == (st1, it1)
