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
