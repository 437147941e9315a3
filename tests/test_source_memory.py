"""The buffers of the particle source belong to solves with a trajectory: a
source-free solve holds the same bytes whatever its patch size, and a sourced
one holds the buffers of two sequences of four steps however large they are
(with fewer, sources are built between the steps instead of beside them)."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(256, 32), (8192, 64)])  # resident, by stage
def test_source_free_solves_hold_no_patches(N, M):
    held = []
    for pts in (64, 512):
        dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
        prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=40 * dt, Fr=5, out_start=0.0,
                         ext_col=N // 2, PTSX=pts, PTSY=pts, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=5.0)
        with bhr.Solver(prm) as s:
            s.step(3)
            free = s.info()["device_bytes"]
            s.set_trajectory(synthetic_plunge(prm.a, dt / 2.0, duration=prm.T + 1.0))
            s.step(20)
            held.append((free, s.info()["device_bytes"]))
            assert np.max(np.abs(s.get_source()[0])) > 0
    assert held[0][0] == held[1][0]
    assert all(sourced - free >= 2 * 2 * 8 * pts * pts for (free, sourced), pts in zip(held, (64, 512)))


@pytest.mark.parametrize("PTSX,PTSY", [(700, 1600), (800, 3000)])
def test_the_largest_patches_are_built_beside_the_steps(PTSX, PTSY):
    prm = bhr.Params(N=256, M=32, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=0.04, T=2.0, Fr=5, out_start=0.0, ext_col=128,
                     PTSX=PTSX, PTSY=PTSY)
    with bhr.Solver(prm) as s:
        free = s.info()["device_bytes"]
        s.set_trajectory(synthetic_plunge(prm.a, prm.dt / 2.0, duration=prm.T + 1.0))
        assert s.info()["device_bytes"] - free >= 2 * 4 * 2 * 8 * PTSX * PTSY
