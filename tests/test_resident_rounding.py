"""Resident steps round as the stage launches do: over thousands of steps their
results drift apart by rounding at random, not by a term that is off the same
way in every stage.

Bounds, with n stages: fields 8 sqrt(n) 2^-53 of their norm -- a random walk
of 64 roundings a stage, the terms of an update that are as large as the field
itself or larger (dissipation, second derivative); waveforms, integrals over
the theta of many points, sqrt(n) 2^-53, the walk of one rounding a stage."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr

pytestmark = pytest.mark.gpu


def evolve(N, M, a, m, steps, tiling, monkeypatch):
    dt = 0.25 * min(400.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-100.0, Xmax=300.0, a=a, m=float(m), dt=dt, T=(steps + 1) * dt, Fr=10, out_start=0.0,
                     ext_col=35 * N // 100, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=20.0, init_width=3.0,
                     init_ell=float(max(2, abs(m))))
    monkeypatch.setenv("BHR_STAGE_TILING", tiling)
    with bhr.Solver(prm) as s:
        assert s.info()["tiling"] == tiling
        s.step(steps)
        return np.stack(s.get_state()), s.waveform()


@pytest.mark.parametrize("a,m", [(0.7, 2), (0.9, 3)])
def test_fields_of_two_row_tiles_drift_by_rounding_only(a, m, monkeypatch):
    steps = 5000
    (u, _), (v, _) = (evolve(896, 176, a, m, steps, tl, monkeypatch) for tl in ("resident", "block8n"))
    bound = 8.0 * np.sqrt(3 * steps) * 2.0 ** -53
    assert np.linalg.norm(u - v) <= bound * np.linalg.norm(v)


@pytest.mark.parametrize("N,M,a,m", [(896, 176, 0.7, 2), (896, 176, 0.9, 3), (1216, 80, 0.7, 2), (1216, 80, 0.3, -1)])
def test_waveforms_drift_by_rounding_only(N, M, a, m, monkeypatch):
    steps = 5000
    (_, (t, h, _)), (_, (t1, h1, _)) = (evolve(N, M, a, m, steps, tl, monkeypatch) for tl in ("resident", "block8n"))
    assert np.array_equal(t, t1)
    assert np.linalg.norm(h - h1) <= np.sqrt(3 * steps) * 2.0 ** -53 * np.linalg.norm(h1)
