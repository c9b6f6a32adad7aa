"""The plain solver's forms -- one thread-block cluster with each way of forming
the quotients, and the cooperative grid -- against the oracle's red-black SOR,
bit for bit (include/physics.hpp:99-157)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (extents, half box): spacings that are powers of two (exact reciprocals), that
# are not (corrected quotients), mixed; one to five planes a block, blocks
# without any, uneven last ones, odd line lengths; grids past the cluster's
# memory (the cooperative form)
CASES = [((32, 32, 32), (16, 16, 16)), ((64, 64, 64), (16, 16, 16)), ((33, 34, 35), (9.3, 8.7, 10.1)),
         ((3, 3, 3), (1.5, 1.1, 2.0)), ((5, 18, 7), (4.1, 5.3, 3.9)), ((50, 61, 40), (10, 9, 8)),
         ((70, 72, 71), (11.3, 10.1, 9.7)), ((80, 78, 82), (12.1, 11.9, 12.3)), ((20, 9, 131), (8, 8, 32.75))]


@pytest.mark.parametrize("n,half", CASES)
@pytest.mark.parametrize("criterion", ["residual", "update"])
def test_plain_solver_is_the_oracles_bit_for_bit(hv, n, half, criterion):
    from hv_b200 import _lib as L
    from hv_oracle import Oracle
    w = hv.CA40_SMALL
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = half[a]
    rng = np.random.default_rng(7)
    G = n[0] * n[1] * n[2]
    rho = np.zeros(2 * G)
    rho[:G] = rng.random(G) * 0.1
    phi = rng.standard_normal(G)
    params = w.run_params()
    if criterion == "update":
        params.sor = L.hv_sor_params(1.5, 1e-4, L.HV_SOR_MAX_UPDATE, 40)
    else:
        params.sor = L.hv_sor_params(1.8, 1e-6, L.HV_SOR_REL_RESIDUAL, 60)
    with hv.Session(world, w.protons, w.neutrons, params, hv.HV_F64) as s:
        s.upload_field(hv.HV_FIELD_DENSITY, rho)
        s.upload_field(hv.HV_FIELD_COULOMB, phi)
        its, metric, ok = s.coulomb_sor(allow_not_converged=True)
        got = s.download_field(hv.HV_FIELD_COULOMB)
    ref = phi.copy()
    # the oracle's order of additions in the residual differs, so its test could
    # fall the other way only within a rounding of the tolerance
    its_o, _ = Oracle(np.float64).sor((n, half), ref, rho, params.sor.omega, params.sor.criterion, params.sor.tol,
                                      params.sor.max_iter)
    assert its == its_o
    assert np.array_equal(got, ref)
