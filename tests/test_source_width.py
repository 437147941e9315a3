"""A patch wider than a block of the source kernel can have threads is refused
by set_trajectory, not by the first step after it."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiling", ["resident", "block8n"])
def test_a_patch_that_is_too_wide_is_refused_by_set_trajectory(tiling, monkeypatch):
    monkeypatch.setenv("BHR_STAGE_TILING", tiling)
    N, M = 256, 32
    dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=40 * dt, Fr=5, out_start=0.0, ext_col=128,
                     PTSX=1024, PTSY=64)
    with bhr.Solver(prm) as s:
        assert s.info()["tiling"] == tiling
        with pytest.raises(bhr.BhrError):
            s.set_trajectory(synthetic_plunge(prm.a, dt / 2.0, duration=prm.T + 1.0))
