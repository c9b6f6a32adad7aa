"""GPU: the pair sums of particles without a finite position, or so far out that
their box has no representable number of cells."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_pair_sums_skip_lost_particles(hv, prec):
    """They are nobody's partner and have none themselves; finite positions so
    far out that their box has no representable number of cells are alone."""
    w = replace(hv.CA40_SMALL, ppn=20)
    dtype, precision = (np.float32, hv.HV_F32) if prec == "f32" else (np.float64, hv.HV_F64)
    base = hv.workload_particles(w, dtype)
    with hv.Session.from_workload(w, precision) as s:
        s.upload_particles(*base)
        s.run(0, hv.HV_PATH_FUSED)
        p = [a.copy() for a in base]
        lost = [0, 1, 2, w.protons]
        for i, v in zip(lost, (np.nan, np.inf, -np.inf, np.nan)):
            p[i % 3][i] = v
        s.upload_particles(*p)
        dp, dn = s.particle_densities()
        far = 1e30 if prec == "f32" else 1e200
        q = [a.copy() for a in base]
        for i, sign in zip(lost, (1, -1, 1, -1)):
            q[i % 3][i] = sign * far
        s.upload_particles(*q)
        fp, fn = s.particle_densities()
        keep = np.setdiff1d(np.arange(base[0].size), lost)
        for a, b in ((dp, fp), (dn, fn)):
            assert np.all(a[lost] == 0.0)
            assert np.all(np.isfinite(a[keep])) and np.all(np.isfinite(b))
            # the same partners, summed in the order of other cells
            assert np.abs(a[keep] - b[keep]).max() <= (1e-5 if prec == "f32" else 1e-13) * np.abs(b).max()
        s.upload_particles(*[np.full_like(a, np.nan) for a in base])
        none_p, none_n = s.particle_densities()
        assert not np.any(none_p) and not np.any(none_n)
