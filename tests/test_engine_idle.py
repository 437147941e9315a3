"""An engine with nothing left to do returns from step() without waiting for
work: the step that finds the last finished solve being released waits for
the release only (a few ms of host work), not for the 200 ms it allows a
solve that is still being prepared."""
import time

import pytest

import bh_ringdown_b200 as bhr

pytestmark = pytest.mark.gpu


def test_last_step_does_not_wait_for_work_that_is_not_there():
    prm = bhr.Params(N=128, M=16, Xmin=-40.0, Xmax=40.0, a=0.3, m=2.0, dt=0.1, Fr=5, T=5.0, out_start=0.0,
                     ext_col=64, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=5.0, init_width=2.0)
    with bhr.Engine() as e:
        e.submit(prm)
        e.run_all()  # first use of the kernels
        spans = []
        for _ in range(3):
            rid = e.submit(prm)
            while e.step(1 << 30):
                t0 = time.perf_counter()
            spans.append(time.perf_counter() - t0)  # the last step() call
            assert e.poll(rid)["state"] == bhr.Engine.DONE
        t0 = time.perf_counter()
        assert e.step(1) == 0  # idle
        spans.append(time.perf_counter() - t0)
    assert min(spans[:3]) < 0.1 and spans[3] < 0.1, spans
