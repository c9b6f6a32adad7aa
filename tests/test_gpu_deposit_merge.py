"""The sorted deposit's merge (k_deposit_merge, csrc/k_plain.cu) bit for bit
against the oracle's sequential deposit, at the edges of its blocks and lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# z extents around a warp (32) and a block (128), and boxes of three nodes a side;
# one particle, a few, and cells of hundreds; particles outside the box and on
# its faces; the spacing 1/2 keeps every cell coordinate's arithmetic alike
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n,particles", [((5, 4, 31), 1), ((5, 4, 32), 7), ((4, 5, 33), 4000), ((3, 3, 3), 5000),
                                         ((3, 6, 127), 3000), ((3, 3, 129), 20000), ((9, 8, 7), 60000)])
def test_merge_keeps_the_sequential_order(hv, n, particles, prec):
    from hv_b200 import _lib as L
    from hv_oracle import Oracle
    dtype = np.float64 if prec == "f64" else np.float32
    half = [0.25 * m for m in n]
    rng = np.random.default_rng(particles)
    protons = particles - particles // 3
    p = [np.ascontiguousarray(rng.uniform(-1.02 * d, 1.02 * d, particles), dtype=dtype) for d in half]
    for c, d in zip(p, half):
        c[:: 11] = dtype(d)
        c[1:: 13] = dtype(-d)
        c[2:: 17] = np.round(4 * c[2:: 17]) / 4
    w = hv.CA40_SMALL
    params = w.run_params()
    params.deposit_mode = hv.HV_DEPOSIT_SORTED
    world = L.hv_world()
    for a in range(3):
        world.n[a], world.d_max[a] = n[a], half[a]
    with hv.Session(world, protons, particles - protons, params, hv.HV_F64 if prec == "f64" else hv.HV_F32) as s:
        s.upload_particles(*p, None, None, None)
        s.deposit()
        got = s.download_field(hv.HV_FIELD_DENSITY_RAW)
    ref = Oracle(dtype).deposit((n, half), protons, particles - protons, *p)
    assert np.array_equal(got, ref)
