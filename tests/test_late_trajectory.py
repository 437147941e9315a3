"""A trajectory set, or replaced, after more steps than set_trajectory makes
records for (8192): the next steps by stage use its records, not what their
place in memory held before.  Against a solve that resumes the checkpoint taken
right after the call, once every record is there; the same launches follow, so
the bits are equal."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replaced", [False, True])
@pytest.mark.parametrize("calls", [(40,), (1, 1, 20)])
def test_a_trajectory_set_late_drives_the_next_steps(replaced, calls, monkeypatch):
    monkeypatch.setenv("BHR_STAGE_TILING", "block8n")
    N, M, late = 128, 16, 8300
    dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=(late + 200) * dt, Fr=10, out_start=0.0,
                     ext_col=80)
    first = synthetic_plunge(prm.a, dt / 2.0, duration=60.0)
    # the same worldline a little further out and heavier: another source on every step
    second = synthetic_plunge(prm.a, dt / 2.0, duration=60.0, r_offset=0.02)
    second[:, 7:9] *= 1.5

    def steps(s):
        out = []
        for n in calls:
            s.step(n)
            out.append(np.stack(s.get_state()))
        return out + list(s.get_source())

    with bhr.Solver(prm) as s:
        if replaced:
            s.set_trajectory(first)
        s.step(late)
        s.set_trajectory(second)
        saved = s.checkpoint()
        got = steps(s)
    with bhr.Solver(prm) as s:
        s.set_trajectory(second)
        s.restore(saved)
        want = steps(s)
    assert np.max(np.abs(want[-2])) > 0
    assert all(np.array_equal(g, w) for g, w in zip(got, want))
