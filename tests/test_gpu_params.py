"""GPU: a change of parameters that is refused leaves the context as it was."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_too_wide_a_stencil_is_refused_as_at_creation(hv):
    """Tap offsets are packed in ten bits: creation refuses a stencil of more
    than 500 nodes, and so does hv_ctx_set_params, before anything changes."""
    from hv_b200 import _lib as L
    world = L.hv_world()
    for a, n in enumerate((600, 8, 8)):
        world.n[a] = n
        world.d_max[a] = 0.05 * n
    w = replace(hv.CA40_SMALL, ppn=10, sigma_r=0.15, deposit_mode=hv.HV_DEPOSIT_SORTED)
    wide = replace(w, sigma_r=13.0, dt=0.1)
    with pytest.raises(hv.HVError) as e:
        hv.Session(world, w.protons, w.neutrons, wide.run_params(), hv.HV_F64)
    assert e.value.status == L.HV_ERR_UNSUPPORTED
    p = hv.workload_particles(w, np.float64)
    out = []
    for refused in (True, False):
        with hv.Session(world, w.protons, w.neutrons, w.run_params(), hv.HV_F64) as s:
            s.upload_particles(*p)
            s.run(2, hv.HV_PATH_FUSED)
            if refused:
                with pytest.raises(hv.HVError) as e:
                    s.set_params(wide.run_params())
                assert e.value.status == L.HV_ERR_UNSUPPORTED
            s.run(2, hv.HV_PATH_FUSED)
            s.deposit()
            s.smooth()
            out.append([s.download_field(hv.HV_FIELD_DENSITY), *s.download_particles()])
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_a_change_of_width_takes_effect(hv):
    """Wider and back: the smoothed density is that of a context created so."""
    w = replace(hv.CA40_SMALL, deposit_mode=hv.HV_DEPOSIT_SORTED)
    p = hv.workload_particles(w, np.float64)
    with hv.Session.from_workload(w, hv.HV_F64) as s:
        s.upload_particles(*p)
        s.run(1, hv.HV_PATH_PLAIN)
        for sigma in (0.9, 0.4, w.sigma_r):
            new = replace(w, sigma_r=sigma)
            s.set_params(new.run_params())
            s.upload_particles(*p)
            s.deposit()
            s.smooth()
            got = s.download_field(hv.HV_FIELD_DENSITY)
            with hv.Session.from_workload(new, hv.HV_F64) as t:
                t.upload_particles(*p)
                t.deposit()
                t.smooth()
                assert np.array_equal(got, t.download_field(hv.HV_FIELD_DENSITY))
            s.run(1, hv.HV_PATH_PLAIN)
