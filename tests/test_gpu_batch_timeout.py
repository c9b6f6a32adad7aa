"""GPU: a batched run in which one instance's solve gives up.

The bounded waits of that instance's solver are set to one poll, so its first
solve runs out and returns (nothing hangs).  The run ends with HV_ERR_TIMEOUT
soon after, and the rows that were good by then are in the caller's buffer."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coarse", [1, 0])
def test_a_timed_out_instance_ends_the_batch_within_two_chunks(hv, coarse):
    from hv_b200 import _lib as L
    from hv_b200.batch import Batch
    w, steps, chunk = hv.PB208_104K, 200, 8
    p = hv.workload_particles(w, np.float32)

    def session(**opts):
        s = hv.Session.from_workload(w, hv.HV_F32)
        s.set_fast_options(sor_coarse=coarse, **opts)
        s.upload_particles(*p)
        s.run(0, hv.HV_PATH_FUSED)
        return s

    with session(sort_every=0) as s:
        alone = s.run(2 * chunk, hv.HV_PATH_FUSED)
        at = s.download_particles()[:3]
    good, bad = session(), session()
    bad.set_fast_options(sor_wait_limit=1)
    obs = np.zeros((2, steps), L.OBS_DTYPE)
    try:
        with Batch([good, bad]) as b:
            st = b.lib.hv_batch_run(b._b, steps, C.c_void_p(obs.ctypes.data))
            assert st == L.HV_ERR_TIMEOUT
            # the other instance's first chunk is there
            d = np.abs(alone["dipole"]).max()
            assert np.abs(obs[0]["dipole"][:chunk] - alone["dipole"][:chunk]).max() <= 1e-4 * d
            assert np.allclose(obs[0]["t"][:chunk], alone["t"][:chunk])
            assert not np.any(obs[1]["sor_iterations"]) and not np.any(obs[1]["t"])
            # and it went at most one chunk further
            for a, q in zip(good.download_particles()[:3], at):
                assert np.abs(a - q).max() <= 1e-2
    finally:
        good.close()
        bad.close()


def test_rows_of_a_long_batch_are_those_of_short_ones(hv):
    """Chunks and a shorter last one, in one call and in three."""
    from hv_b200.batch import Batch
    from dataclasses import replace
    w = replace(hv.CA40_SMALL, ppn=40, deposit_mode=hv.HV_DEPOSIT_SORTED)
    p = hv.workload_particles(w, np.float32)
    out = []
    for parts in ((45,), (16, 8, 21)):
        sessions = [hv.Session.from_workload(w, hv.HV_F32) for _ in range(3)]
        for s in sessions:
            s.upload_particles(*p)
        try:
            with Batch(sessions) as b:
                out.append(np.concatenate([b.run(k) for k in parts], axis=1))
        finally:
            for s in sessions:
                s.close()
    assert np.allclose(out[0]["t"], np.arange(45) * w.dt)
    assert np.all(out[0]["sor_iterations"] >= 1)
    d = np.abs(out[0]["dipole"]).max()
    # a call's end closes the kick and the next one reads the same state
    assert np.abs(out[0]["dipole"] - out[1]["dipole"]).max() <= 1e-5 * d
