"""GPU: the direct Coulomb solve eliminates along x from both ends, so a source
mirrored in x has the mirrored solution, bit for bit.

With an odd number of planes the two sides meet in a middle node that both of
them compute: the result must not depend on which side's value is kept."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _position(t, n, d_max):
    """A float position whose grid coordinate (n / 2) (x / d_max + 1) is t
    exactly in float, or None."""
    x0 = F((2.0 * t / n - 1.0) * d_max)
    for k in range(-40, 41):
        x = x0
        for _ in range(abs(k)):
            x = np.nextafter(x, F(np.inf if k > 0 else -np.inf))
        if F(F(n) / F(2)) * F(F(x / F(d_max)) + F(1)) == F(t):
            return x
    return None


@pytest.mark.parametrize("n", [(33, 20, 24), (5, 12, 11), (34, 20, 24), (129, 40, 33)])
def test_mirrored_source_has_the_mirrored_solution(hv, n):
    """The deposited cells are exact in float, the smoothing stencil is the
    node itself, the faces are zero and the solve starts from zero, so the two
    right-hand sides are mirror images bit for bit; after one correction phi is
    the correction itself."""
    from dataclasses import replace

    from hv_b200 import _lib as L
    world = L.hv_world()
    for a in range(3):
        world.n[a] = n[a]
        world.d_max[a] = 0.5 * n[a]
    rng = np.random.default_rng(1)
    pairs = []
    while len(pairs) < 200:
        t = rng.integers(64, 64 * (n[0] - 2)) / 64.0
        x = _position(t, n[0], world.d_max[0]), _position(n[0] - 1 - t, n[0], world.d_max[0])
        if x[0] is not None and x[1] is not None:
            pairs.append(x)
    m = len(pairs)
    rest = [rng.uniform(-0.8 * world.d_max[a], 0.8 * world.d_max[a], m).astype(F) for a in (1, 2)]
    w = replace(hv.CA40_SMALL, sigma_r=0.2, sor_max_iter=1, deposit_mode=hv.HV_DEPOSIT_SORTED)
    params = w.run_params()
    params.z, params.n, params.part_per_nucleon = 0, 1, 1
    phi = []
    for side in (0, 1):
        with hv.Session(world, m, 0, params, hv.HV_F32) as s:
            s.upload_particles(np.array([p[side] for p in pairs], F), *rest, *[np.zeros(m, F)] * 3)
            s.run(0, hv.HV_PATH_FUSED)
            phi.append((s.download_field(hv.HV_FIELD_DENSITY)[:s.G].reshape(n),
                        s.download_field(hv.HV_FIELD_COULOMB).reshape(n)))
    assert np.array_equal(phi[1][0], phi[0][0][::-1]) and phi[0][0].max() > 0.0
    assert np.array_equal(phi[1][1], phi[0][1][::-1]), np.abs(phi[1][1] - phi[0][1][::-1]).max()
    assert phi[0][1].max() > 0.0


def test_odd_extents_repeat_bit_for_bit(hv):
    """The reproducible mode on odd planes: two sessions give the same bits."""
    from dataclasses import replace
    w = replace(hv.CA40_SMALL, n=33, deposit_mode=hv.HV_DEPOSIT_SORTED)
    out = []
    for _ in range(2):
        with hv.Session.from_workload(w, hv.HV_F32) as s:
            s.upload_particles(*hv.workload_particles(w, F))
            s.run(12, hv.HV_PATH_FUSED)
            out.append([*s.download_particles(), s.download_field(hv.HV_FIELD_COULOMB)])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
