"""The two-launch smoothing of the fused float path (k_smooth_discs,
k_smooth_planes) and the Skyrme potential it writes, against the direct tap sum
and potential in double on the same raw density."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# extents around the 16 x 16 tiles (one short, exact, one past, several), half
# widths 1 to 16, unequal spacings, and density that reaches the faces
@pytest.mark.parametrize("n,half", [((15, 16, 17), (9, 9, 9)), ((33, 34, 35), (9, 10, 11)), ((75, 61, 50), (10, 9, 8)),
                                    ((12, 48, 31), (5, 9, 6)), ((20, 20, 20), (3, 3, 3)), ((5, 3, 40), (9, 9, 9)),
                                    ((98, 96, 97), (8, 8, 8)), ((40, 130, 20), (9, 8, 9))])
def test_disc_smoothing_and_potential_match_the_direct_double_sums(hv, n, half):
    """Float sums of non-negative terms in three nested levels (z-runs of up to
    17 pairs, discs of 17, planes of 33): relative rounding below 70 * 2^-24 =
    4.2e-6 of the result's own size, hence of the maximum.  The potential's
    terms A t and B t^gamma (both below 500 MeV at the densities here) carry
    that density error, t^gamma by the fast power (2^-21 of its value) too."""
    from hv_b200 import _lib as L
    w = hv.CA40_SMALL
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = half[a]
    p = hv.workload_particles(w, np.float32)
    with hv.Session(world, w.protons, w.neutrons, w.run_params(), hv.HV_F32) as s:
        s.upload_particles(*p)
        s.run(0, hv.HV_PATH_FUSED)
        raw = s.download_field(hv.HV_FIELD_DENSITY_RAW)
        rho = s.download_field(hv.HV_FIELD_DENSITY)
        U = s.download_field(hv.HV_FIELD_POTENTIAL)
        phi = s.download_field(hv.HV_FIELD_COULOMB)
    with hv.Session(world, w.protons, w.neutrons, w.run_params(), hv.HV_F64) as s:
        s.upload_field(hv.HV_FIELD_DENSITY_RAW, raw.astype(np.float64))
        s.smooth()
        ref = s.download_field(hv.HV_FIELD_DENSITY)
        s.skyrme()
        ref_u = s.download_field(hv.HV_FIELD_POTENTIAL)
    assert np.abs(rho - ref).max() <= 4.2e-6 * ref.max()
    g = n[0] * n[1] * n[2]
    ref_u[:g] += phi
    A, B, C, gamma = w.skyrme()
    t = (ref[:g] + ref[g:]).max() / 0.16
    scale = abs(A) * t + B * t ** gamma + 2 * C * t
    bound = scale * (4.2e-6 * (1 + gamma) + 2.0 ** -21) + 2.0 ** -22 * np.abs(phi).max()
    assert np.abs(U - ref_u).max() <= bound
