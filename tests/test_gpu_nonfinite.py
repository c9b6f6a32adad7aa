"""GPU: a fused solve that is not finite is reported on every step.

One interior node of the Coulomb potential is set to NaN through the host API
between two runs.  No later solve can meet the stopping rule (its first
residual is NaN already), so every later row carries
HV_OBS_SOR_NOT_CONVERGED and no row claims zero iterations.  Particles that
reach NaN positions are outside the grid for every kernel."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _poison(hv, s, n):
    phi = s.download_field(hv.HV_FIELD_COULOMB)
    phi.reshape(n, n, n)[n // 2, n // 2, n // 2] = np.nan
    s.upload_field(hv.HV_FIELD_COULOMB, phi)


# the direct solve and the sweeps, float and double, both stopping rules
FORMS = [("f32", 1e-6, {}), ("f32", 1e-6, dict(sor_coarse=0)),
         ("f32", 1e-6, dict(sor_exchange=1)), ("f64", 1e-11, {}), ("f64", 1e-6, {}), ("f32", None, {})]


@pytest.mark.parametrize("prec,tol,opts", FORMS)
def test_non_finite_solves_are_flagged_on_every_step(hv, prec, tol, opts):
    w = hv.CA40_SMALL.with_reference_sor() if tol is None else replace(hv.CA40_SMALL, sor_tol=tol)
    dtype, precision = (np.float32, hv.HV_F32) if prec == "f32" else (np.float64, hv.HV_F64)
    with hv.Session.from_workload(w, precision) as s:
        s.set_fast_options(**opts)
        s.upload_particles(*hv.workload_particles(w, dtype))
        first = s.run(2, hv.HV_PATH_FUSED)
        _poison(hv, s, w.n)
        obs = s.run(5, hv.HV_PATH_FUSED)
    assert not np.any(first["flags"] & 1)
    assert np.all(obs["flags"] & 1), obs["flags"]
    assert np.all(obs["sor_iterations"] >= 1), obs["sor_iterations"]


@pytest.mark.parametrize("coarse", [1, 0])
def test_a_non_finite_instance_of_a_batch_is_flagged_alone(hv, coarse):
    from hv_b200.batch import Batch
    w = hv.CA40_SMALL
    sessions = []
    for _ in range(2):
        s = hv.Session.from_workload(w, hv.HV_F32)
        s.set_fast_options(sor_coarse=coarse)
        s.upload_particles(*hv.workload_particles(w, np.float32))
        sessions.append(s)
    try:
        with Batch(sessions) as b:
            b.run(2)
            _poison(hv, sessions[1], w.n)
            obs = b.run(5)
    finally:
        for s in sessions:
            s.close()
    assert not np.any(obs[0]["flags"] & 1)
    assert np.all(obs[1]["flags"] & 1), obs[1]["flags"]
    assert np.all(obs[1]["sor_iterations"] >= 1)
