"""Stages of grids and of batches whose states do not stay in L2 walk the
tiles forward and backward in turn (block8n).  A tile's result does not depend
on the order, so the fields agree with the 256-thread tiles', which always walk
forward, to rounding (fields 1e-13 of scale, waveforms relative L2 1e-12),
through eager steps, single-step graphs and 16-step graphs, at a size just
above the threshold, for SSP-RK3 and classical RK4."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

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


def test_turning_mixed_stages_match_one_way_stages(monkeypatch):
    """Mixed precision above the size from which the FP32 stages turn too.
    The FP64 stage's tilings agree to rounding, so its FP32 correction (dt L u,
    1e-2 of u and less) moves by an FP32 rounding, 6e-8, at most: 1e-8 of scale
    over the run."""
    N, M = 8192, 176
    prm = bhr.Params(N=N, M=M, Xmin=-100.0, Xmax=300.0, a=0.8, m=2.0, dt=0.25 * min(400.0 / N, 1.6 * np.pi / M), T=10.0,
                     Fr=4, out_start=0.0, ext_col=N * 32 // 100, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=25.0,
                     init_width=3.0, precision=bhr.BHR_MIXED)
    out = []
    for tiling, split in (("block8", (1, 2, 38)), ("block8n", (1, 2, 38)), ("block8n", (41,))):
        monkeypatch.setenv("BHR_STAGE_TILING", tiling)
        with bhr.Solver(prm) as s:
            for n in split:
                s.step(n)
            out.append(s.get_state())
    scale = max(np.max(np.abs(f)) for f in out[0])
    assert max(np.max(np.abs(a - b)) for a, b in zip(out[0], out[1])) <= 1e-8 * scale
    assert all(np.array_equal(a, b) for a, b in zip(out[1], out[2]))


def test_a_turning_batch_gives_the_rows_of_the_solves_alone():
    """A batch large enough to turn, of FP64 and mixed solves and a plunge of
    different lengths (the last ones run on without turning): every request
    bit-identical to the same one alone, which does not turn."""
    def request(N, M, m, T, precision=bhr.BHR_FP64, traj=False):
        dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
        prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=m, dt=dt, T=T, Fr=3, out_start=0.0,
                         ext_col=N * 6 // 10, init_kind=0 if traj else bhr.BHR_INIT_GAUSSIAN, init_center=10.0,
                         init_width=2.0, precision=precision)
        return prm, synthetic_plunge(prm.a, dt / 2.0, duration=T) if traj else None

    reqs = [request(4096, 128, 2.0, 0.3), request(2048, 128, -1.0, 0.5, bhr.BHR_MIXED),
            request(2048, 160, 2.0, 0.4, traj=True), request(1024, 64, 3.0, 0.6), request(2048, 128, 1.0, 0.25)]
    assert sum(p.N * p.M for p, _ in reqs) * 96 >= 96 << 20

    def rows(some):
        with bhr.Engine() as e:
            ids = [e.submit(p, t) for p, t in some]
            e.run_all()
            return [e.result(i) for i in ids]

    for (alone,), together in zip([rows([r]) for r in reqs], rows(reqs)):
        assert len(alone[0]) > 3
        for x, y in zip(alone, together):
            assert np.array_equal(x, y)
