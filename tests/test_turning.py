"""Stages of grids whose states do not stay in L2 walk the tiles forward and
backward in turn (block8n).  A tile's result does not depend on the order, so
the fields agree with the 256-thread tiles', which always walk forward, to
rounding (fields 1e-13 of scale, waveforms relative L2 1e-12), through eager
steps, single-step graphs and 16-step graphs, at a size just above the
threshold, for SSP-RK3 and classical RK4."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,integrator", [(8192, 128, bhr.BHR_SSPRK3), (7168, 112, bhr.BHR_RK4)])
def test_turning_stages_match_one_way_stages(N, M, integrator, monkeypatch):
    prm = bhr.Params(N=N, M=M, Xmin=-100.0, Xmax=300.0, a=0.8, m=2.0, dt=0.25 * min(400.0 / N, 1.6 * np.pi / M), T=50.0,
                     Fr=4, out_start=0.0, ext_col=N * 32 // 100, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=25.0,
                     init_width=3.0, integrator=integrator)
    out = []
    for tiling in ("block8", "block8n"):
        monkeypatch.setenv("BHR_STAGE_TILING", tiling)
        with bhr.Solver(prm) as s:
            assert s.info()["tiling"] == tiling
            for n in (1, 2, 38):
                s.step(n)
            out.append((s.get_state(), s.waveform()))
    (f0, w0), (f1, w1) = out
    scale = max(np.max(np.abs(f)) for f in f0)
    assert max(np.max(np.abs(a - b)) for a, b in zip(f0, f1)) <= 1e-13 * scale
    assert np.array_equal(w0[0], w1[0]) and len(w0[0]) == 11
    assert np.linalg.norm(w0[1] - w1[1]) <= 1e-12 * np.linalg.norm(w0[1])
