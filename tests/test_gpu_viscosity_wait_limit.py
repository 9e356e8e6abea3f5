"""The CTAs of a viscosity bottom cycle or coarsest solve wait for one another
within a limit.  With a limit of 0 every wait gives up: the kernels still end,
the call fails, and other handles solve as before.  16^3: the coarsest CG in
one CTA; 24^3: over eight."""
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


def make(n):
    from uaamg_b200.viscosity import L_with_level, simd_viscosity3d
    sc = scenes.plain_viscosity_scene(n=n, seed=2)
    lv = L_with_level.create_viscosity_matrix(sc.viscosity, sc.liquid_phi, sc.solid_phi, sc.dt, sc.rho, sc.dx)
    return lv, simd_viscosity3d(lv), lv.build_rhs(sc.u, sc.v, sc.w, sc.solid_velocity)


@pytest.mark.parametrize("graph", [0, 2])
@pytest.mark.parametrize("n", [16, 24])
def test_a_wait_that_gives_up_fails_the_solve(gpu, monkeypatch, n, graph):
    from uaamg_b200._lib import UaamgError
    lv, s, rhs = make(n)
    s.use_graph = graph
    want = np.zeros_like(rhs)
    st = s.pcg_solve(want, 1e-6, rhs)  # (100 iterations from zero may or may not reach the tolerance)
    assert np.isfinite(want).all() and want.any()
    monkeypatch.setenv("UAAMG_VISC_WAIT_US", "0")
    lv0, s0, _ = make(n)
    s0.use_graph = graph
    for _ in range(2):
        with pytest.raises(UaamgError, match="waited too long"):
            s0.pcg_solve(np.zeros_like(rhs), 1e-6, rhs)
    monkeypatch.delenv("UAAMG_VISC_WAIT_US")
    lv1, s1, _ = make(n)
    for t in (s, s1):
        x = np.zeros_like(rhs)
        assert t.pcg_solve(x, 1e-6, rhs) == st and np.array_equal(x, want)


@pytest.mark.parametrize("n", [16, 24])
def test_calls_outside_a_solve_report_it(gpu, monkeypatch, n):
    from uaamg_b200._lib import UaamgError
    lv, s, rhs = make(n)
    r = np.ones_like(rhs)
    z, b = s.precondition(r), np.ones((3, lv.leaf_count(lv.num_levels() - 1), 512), np.float32)
    x = lv.solve_exact(b)
    monkeypatch.setenv("UAAMG_VISC_WAIT_US", "0")
    lv0, s0, _ = make(n)
    with pytest.raises(UaamgError, match="waited too long"):
        s0.precondition(r)
    if n == 24:
        with pytest.raises(UaamgError, match="waited too long"):
            lv0.solve_exact(b)
    else:  # one CTA: nothing to wait for, and the error of the call before is not this one's
        assert np.array_equal(lv0.solve_exact(b), x)
    assert np.array_equal(s.precondition(r), z) and np.array_equal(lv.solve_exact(b), x)
