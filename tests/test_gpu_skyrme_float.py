"""The float fused path's Skyrme potential (csrc/skyrme.cuh) against NumPy's in
double on the same smoothed density."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the potential written by the smoothing (32^3, 30 x 31 x 29) and by its own
# kernel (128^3: four nodes a thread behind the FFT smoothing)
@pytest.mark.parametrize("n,h", [((32, 32, 32), 1.0), ((30, 31, 29), 0.9), ((128, 128, 128), 0.25)])
@pytest.mark.parametrize("sigma", [1.0 / 6.0, 0.5, 1.0])
def test_float_potential_is_the_double_one_rounded_once(hv, n, h, sigma):
    """Neutrons' U = A t + B t^gamma + 2 C (rho_n - rho_p) / rho_0.  From t =
    2^-8 on it is formed in double (power within 1e-9) and rounded to float
    once: 2^-24 of |U|, to which come 1e-9 of the power's term and 2^-50 of the
    sums.  Below, three float products and sums of terms no larger than |A| t +
    B t^gamma + 2 C t (4 * 2^-24 of them) and the fast power, 2^-20 of its term.
    The boundary itself is rounded in float: both bounds hold near it."""
    from dataclasses import replace

    from hv_b200 import _lib as L
    w = replace(hv.CA40_SMALL, sigma=sigma)
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = 0.5 * n[a] * h
    with hv.Session(world, w.protons, w.neutrons, w.run_params(), hv.HV_F32) as s:
        s.upload_particles(*hv.workload_particles(w, np.float32))
        s.run(0, hv.HV_PATH_FUSED)
        rho = s.download_field(hv.HV_FIELD_DENSITY).astype(np.float64)
        U = s.download_field(hv.HV_FIELD_POTENTIAL)
    g = n[0] * n[1] * n[2]
    A, B, C, gamma = w.skyrme()
    rp, rn = rho[:g], rho[g:]
    t = (rp + rn) / 0.16
    power = np.abs(B) * t ** gamma
    ref = A * t + B * t ** gamma + 2.0 * C * (rn - rp) / 0.16
    size = np.abs(A) * t + power + 2.0 * np.abs(C) * t
    near = 2.0 ** -24 * np.abs(ref) + 1e-9 * power + 2.0 ** -50 * size
    far = 4 * 2.0 ** -24 * size + 2.0 ** -20 * power
    edge = 2.0 ** -8
    assert t.max() > 0.5 and np.any((t > 0) & (t < edge))
    bound = np.where(t > edge * (1 + 1e-6), near, np.maximum(near, far))
    assert np.all(np.abs(U[g:] - ref) <= bound)
