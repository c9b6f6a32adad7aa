"""The fused path's direct Coulomb solve (k_poisson.cu) against a double
solution of the same discrete equation: the reference's 7-point operator with
monopole faces (include/physics.hpp:99-157, include/tools.hpp:283-300), solved
by sine transforms in NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALF_BOX = (10.0, 9.0, 11.0)


def _world(n):
    from hv_b200 import _lib as L
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = HALF_BOX[a]
    return world


def exact_phi(n, Z, rho_p):
    """phi of the discrete problem in double: faces at 1.44 Z / r, the interior
    by the orthonormal sine transform of each axis."""
    h = [2.0 * d / m for d, m in zip(HALF_BOX, n)]
    pos = [d * (2.0 * np.arange(m) / m - 1.0) for d, m in zip(HALF_BOX, n)]
    r = np.sqrt(pos[0][:, None, None] ** 2 + pos[1][None, :, None] ** 2 + pos[2][None, None, :] ** 2)
    phi = np.zeros(n)
    face = np.ones(n, bool)
    face[1:-1, 1:-1, 1:-1] = False
    phi[face] = 1.44 * Z / r[face]
    b = 4.0 * np.pi * 1.44 * rho_p.astype(np.float64)
    for a in range(3):
        b = b + (np.roll(phi, 1, a) + np.roll(phi, -1, a)) / h[a] ** 2
    f = b[1:-1, 1:-1, 1:-1]
    lam = 0.0
    S = []
    for a, m in enumerate(n):
        k = np.arange(1, m - 1)
        S.append(np.sin(np.pi * np.outer(k, k) / (m - 1)) * np.sqrt(2.0 / (m - 1)))
        shape = [1, 1, 1]
        shape[a] = -1
        lam = lam + ((2.0 - 2.0 * np.cos(np.pi * k / (m - 1))) / h[a] ** 2).reshape(shape)

    def transform(g):
        for a in range(3):
            g = np.moveaxis(np.tensordot(S[a], g, axes=([1], [a])), 0, a)
        return g

    phi[1:-1, 1:-1, 1:-1] = transform(transform(f) / lam)
    return phi


# edges of the forms: one interior node, odd and even halves, extents off the
# tiles' multiples, the two row tiles and the two-tile form, matrices shared
# between y and z or not, reloaded matrices, long and short x
SHAPES = [(3, 3, 3), (4, 5, 6), (32, 32, 32), (33, 34, 35), (64, 64, 64), (75, 61, 50), (61, 75, 50), (63, 66, 67),
          (128, 128, 128), (20, 127, 128), (16, 126, 131), (12, 150, 150), (6, 160, 170), (200, 16, 16), (17, 9, 130)]


@pytest.mark.parametrize("n", SHAPES)
def test_direct_solve_matches_the_double_solution(hv, n):
    """With the rule at 1e-10 the solve's own error is far below float: the
    downloaded float phi is the exact solution of the downloaded density to
    the rounding of the two floats involved (2 x 2^-24 of the largest value),
    after the first solve and after steps from each starting guess; and one or
    two corrections a step are the direct form's count."""
    from dataclasses import replace
    w = replace(hv.CA40_SMALL, sor_tol=1e-10, dt=0.25)
    p = hv.workload_particles(w, np.float32)
    for guess in (hv.HV_WARM_PREVIOUS, hv.HV_WARM_QUADRATIC):
        with hv.Session(_world(n), w.protons, w.neutrons, w.run_params(), hv.HV_F32) as s:
            s.set_fast_options(sor_warm_start=guess)
            s.upload_particles(*p)
            for steps in (0, 4):
                obs = s.run(steps, hv.HV_PATH_FUSED)
                rho = s.download_field(hv.HV_FIELD_DENSITY).reshape(2, *n)
                phi = s.download_field(hv.HV_FIELD_COULOMB).reshape(n)
                ref = exact_phi(n, w.Z, rho[0])
                err = np.abs(phi - ref).max() / np.abs(ref).max()
                assert err < 1.2e-7, (n, guess, steps, err)
            assert not np.any(obs["flags"] & 1)
            assert np.all(obs["sor_iterations"] <= 3), obs["sor_iterations"]


def test_direct_solve_stops_at_the_iteration_cap(hv):
    """max_iter corrections at most, flagged when they do not meet the rule."""
    from dataclasses import replace
    w = replace(hv.CA40_SMALL, sor_tol=1e-13, sor_max_iter=1)
    p = hv.workload_particles(w, np.float32)
    with hv.Session.from_workload(w, hv.HV_F32) as s:
        s.upload_particles(*p)
        obs = s.run(2, hv.HV_PATH_FUSED)
    assert np.all(obs["sor_iterations"] == 1)
    assert np.all(obs["flags"] & 1)


@pytest.mark.parametrize("n", [(3, 4, 5), (32, 32, 32), (75, 61, 50), (64, 64, 64), (20, 127, 128)])
def test_direct_double_solve_matches_the_double_solution(hv, n):
    """A double context with a rule of 1e-11 takes the direct form.  The solve
    leaves |r|_2 <= 1e-11 |b|_2, so phi is off by at most |r|_2 over the
    smallest eigenvalue (and a few roundings of phi)."""
    from dataclasses import replace
    tol = 1e-11
    w = replace(hv.CA40_SMALL, sor_tol=tol, dt=0.25)
    p = hv.workload_particles(w, np.float64)
    lam = sum((2.0 - 2.0 * np.cos(np.pi / (m - 1))) * (m / (2.0 * d)) ** 2 for m, d in zip(n, HALF_BOX))
    with hv.Session(_world(n), w.protons, w.neutrons, w.run_params(), hv.HV_F64) as s:
        s.upload_particles(*p)
        for steps in (0, 4):
            obs = s.run(steps, hv.HV_PATH_FUSED)
            rho = s.download_field(hv.HV_FIELD_DENSITY).reshape(2, *n)
            phi = s.download_field(hv.HV_FIELD_COULOMB).reshape(n)
            ref = exact_phi(n, w.Z, rho[0])
            b = 4.0 * np.pi * 1.44 * np.linalg.norm(rho[0][1:-1, 1:-1, 1:-1])
            assert np.abs(phi - ref).max() < tol * b / lam + 1e-13 * np.abs(ref).max(), (n, steps)
        assert not np.any(obs["flags"] & 1)
        assert np.all(obs["sor_iterations"] <= 5), obs["sor_iterations"]


def test_direct_adjoint_solve_does_not_depend_on_the_objective_scale(hv):
    """The transposed solves' correction is in float on values scaled to their
    largest source: the gradient of an objective scaled by 2^-140 (below
    float's range) is the scaled gradient, and no solve stops unconverged."""
    from dataclasses import replace

    from hv_b200.adjoint import AdjointRun
    steps = 6
    w = replace(hv.CA40_SMALL, ppn=40, sor_tol=1e-12, deposit_mode=hv.HV_DEPOSIT_SORTED)
    p = hv.workload_particles(w, np.float64)
    wts = np.random.default_rng(3).standard_normal(steps)
    run = AdjointRun(w, p, steps, checkpoint_every=3, path=hv.HV_PATH_FUSED)
    try:
        run.forward((w.t0, w.t3, w.sigma, w.a_sym))
        g1 = run.backward(wts)
        g2 = run.backward(wts * 2.0 ** -140)
        _, its, unconverged = run.session.adjoint_stats()
    finally:
        run.close()
    assert unconverged == 0 and 0 < its <= 6 * (steps + 1)
    # each solve's own tolerance, 1e-12, is all that may differ
    assert np.max(np.abs(g2 * 2.0 ** 140 - g1)) <= 1e-9 * np.abs(g1).max()
