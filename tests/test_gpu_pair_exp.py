"""The double pair sums' exponential (csrc/pdens.cu: by table, Tang 1989)
against NumPy's over its whole range [0, 8], through hv_particle_densities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pair_exponential_matches_numpy_over_the_cutoff_sphere(hv):
    """Two particles at distance d give each other exp(-d^2 / 2 sigma_r^2) on
    top of their own 1; 4000 such pairs, far apart from each other, cover
    d^2 / 2 sigma_r^2 in [0, 8].  d^2 and its exponent are rounded three times
    (relative 2^-53 each, at most 8 * 3 * 1.1e-16 in the exponent), the table's
    exponential adds at most 4e-16 relative, the sums and the normalisation
    1e-15 of 1."""
    from dataclasses import replace
    pairs = 4000
    w = replace(hv.CA40_SMALL, Z=2, N=0, ppn=pairs)
    assert w.particles == 2 * pairs
    t = np.linspace(0.0, 7.999999, pairs)
    d = np.sqrt(2.0 * t) * w.sigma_r
    x = np.repeat(10.0 * np.arange(pairs), 2)
    z = np.zeros(2 * pairs)
    z[1::2] = d
    zero = np.zeros(2 * pairs)
    with hv.Session.from_workload(w, hv.HV_F64) as s:
        s.upload_particles(x, zero, z, zero, zero, zero)
        dp, dn = s.particle_densities()
    term = 1.0 / (pairs * (2.0 * np.pi * w.sigma_r ** 2) ** 1.5)
    ref = 1.0 + np.exp(-(d * d) * (1.0 / (2.0 * w.sigma_r ** 2)))
    got = dp / term
    bound = np.exp(-t) * (24 * 1.2e-16 + 4e-16) + 2e-15
    assert np.all(np.abs(got.reshape(-1, 2) - ref[:, None]) <= bound[:, None])
    assert np.all(dn == 0.0)
