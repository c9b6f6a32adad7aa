"""GPU: the autotuners look only at choices that the solve has."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coarse", [1, 0])
def test_autotune_searches_tiles_for_sweeps_only(hv, coarse):
    """Twelve particle configurations; then one timing of a direct solve, or
    the sweeps' tiles.  The report describes the solve that runs."""
    w = hv.PB208_104K
    trial = 1
    with hv.Session.from_workload(w, hv.HV_F32) as s:
        s.set_fast_options(sor_coarse=coarse)
        s.upload_particles(*hv.workload_particles(w, np.float32))
        rep = s.autotune(trial)
        t = s.run(1, hv.HV_PATH_FUSED)["t"][0]
    # an untimed and the timed steps of every configuration
    assert np.isclose(t, rep["candidates"] * (1 + trial) * w.dt, rtol=1e-6)
    assert rep["sor_ms"] > 0.0
    if coarse:
        assert rep["candidates"] == 13, rep
        assert rep["sor_tile_rank"] == 0
        # whole planes, one per block
        assert rep["sor_rows"] == w.n and rep["sor_planes"] == -(-(w.n - 2) // rep["sor_blocks"])
    else:
        assert 13 <= rep["candidates"] <= 16
        # a tile of some rows of some planes covers the interior planes
        assert rep["sor_planes"] * rep["sor_rows"] * rep["sor_blocks"] >= (w.n - 2) * w.n


@pytest.mark.parametrize("coarse", [(1, 1), (0, 1), (0, 0)])
def test_batch_autotune_searches_caps_for_sweeps_only(hv, coarse):
    """Three block sizes of the particle step, and six caps before them where
    an instance of the batch sweeps."""
    from hv_b200.batch import Batch
    w = hv.CA40_SMALL
    trial = 1
    sessions = []
    for c in coarse:
        s = hv.Session.from_workload(w, hv.HV_F32)
        s.set_fast_options(sor_coarse=c)
        s.upload_particles(*hv.workload_particles(w, np.float32))
        sessions.append(s)
    try:
        with Batch(sessions) as b:
            cap = b.autotune(trial)
            tiles = b.tiles()
            obs = b.run(1)
    finally:
        for s in sessions:
            s.close()
    trials = 3 if all(coarse) else 9
    assert np.allclose(obs["t"][:, 0], trials * (1 + trial) * w.dt)
    assert cap == 0 if all(coarse) else cap in (0, 64, 32, 16, 8, 4)
    for c, (planes, rows, blocks, _) in zip(coarse, tiles):
        if c:
            assert rows == w.n and planes == -(-(w.n - 2) // blocks)
