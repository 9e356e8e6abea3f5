"""Viscosity that varies in part of the domain: few or none of level 0's leaves
are plain, and which passes take them apart depends on how many there are
(csrc/viscosity_plain.h).  Whatever the choice, the preconditioner and a whole
solve equal those of the general passes, and of the lists in every pass, bit
for bit."""
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


# side, part of the domain that varies: every pass with lists; the colours only; the colours only, few plain leaves; none
@pytest.mark.parametrize("n,part", [(128, 0.25), (128, 0.6), (104, 0.8), (91, 1.0)])
def test_forms_equal(gpu, monkeypatch, n, part):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.plain_viscosity_scene(n=n, seed=1)
    c = (np.arange(n) + 0.5) / n
    X, Y, Z = np.meshgrid(c, c, c, indexing="ij")
    mu = np.where(X < part, 1e3 * np.exp(0.8 * np.sin(7 * (X - part)) * np.cos(5 * Y + 3 * Z)), 1e3)
    visc = dense_to_leaves(mu.astype(np.float32), background=np.float32(1e3))
    out = []
    for leaves in (None, str(2**31 - 1), "1024"):
        if leaves:
            monkeypatch.setenv("UAAMG_VISC_PLAIN_LEAVES", leaves)
        lv = L_with_level.create_viscosity_matrix(visc, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
        assert lv.leaf_count(0) >= 1024
        rhs = lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)
        x = lv.gather_velocity(sc.u, sc.v, sc.w)
        s = simd_viscosity3d(lv)
        z = s.precondition(rhs)
        st = s.pcg_solve(x, 1e-6, rhs)
        out.append((z, x, st, s.m_iteration))
    for z, x, st, it in out[1:]:
        assert (st, it) == out[0][2:] and st == 0
        assert np.array_equal(z, out[0][0]) and np.array_equal(x, out[0][1])
