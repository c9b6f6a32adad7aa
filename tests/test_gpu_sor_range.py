"""GPU: the plain solver's quotients over the whole range of a double, against
the oracle's divisions bit for bit (include/physics.hpp:99-157): potentials so
small or large that the corrected quotient's remainders would not be exact, and
exact zeros of both signs among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# extents of the cluster form and of the cooperative one; no spacing squares to
# a power of two
@pytest.mark.parametrize("n,half", [((33, 34, 35), (9.3, 8.7, 10.1)), ((80, 78, 82), (12.1, 11.9, 12.3)),
                                    ((300, 9, 10), (40.0, 1.3, 1.4))])
@pytest.mark.parametrize("scale", [1.0, 1e-281, 1e-295, 1e-307, 1e-316, 1e281, 1e300])
def test_plain_solver_divides_exactly_at_any_scale(hv, n, half, scale):
    from hv_b200 import _lib as L
    from hv_oracle import Oracle
    w = hv.CA40_SMALL
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = half[a]
    rng = np.random.default_rng(11)
    G = n[0] * n[1] * n[2]
    phi = rng.standard_normal(G) * scale
    phi[rng.random(G) < 0.1] = 0.0
    phi[rng.random(G) < 0.1] = -0.0
    params = w.run_params()
    params.sor = L.hv_sor_params(1.5, 5e-324, L.HV_SOR_MAX_UPDATE, 4)
    with hv.Session(world, w.protons, w.neutrons, params, hv.HV_F64) as s:
        s.upload_field(hv.HV_FIELD_DENSITY, np.zeros(2 * G))
        s.upload_field(hv.HV_FIELD_COULOMB, phi)
        its, _, _ = s.coulomb_sor(allow_not_converged=True)
        got = s.download_field(hv.HV_FIELD_COULOMB)
    ref = phi.copy()
    its_o, _ = Oracle(np.float64).sor((n, half), ref, np.zeros(2 * G), 1.5, L.HV_SOR_MAX_UPDATE, 5e-324, 4)
    assert its == its_o == 4
    assert np.all(np.isfinite(ref))
    assert np.array_equal(got.view(np.int64), ref.view(np.int64)), np.sum(got != ref)
