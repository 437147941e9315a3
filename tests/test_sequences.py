"""Steps run in sequences of up to 16: their stages follow one another, the
previous sequence is extracted and the next one's sources are built beside
them.  However a run is split into calls -- single steps, sequences that are
not full, full ones and remainders, captured (small grids) or launched
directly -- the fields are the same bits, and the waveform (integrated and
projected per sequence or per step) agrees to rounding (relative L2 1e-13),
with an interior extraction column and ones that are closure points, a source,
mixed precision, RK4, tilings that record the extraction column themselves and
ones that do not, and patches so large that a sequence is one step."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

pytestmark = pytest.mark.gpu

SPLITS = [[1] * 53, [53], [2, 15, 16, 17, 3], [48, 1, 4]]


@pytest.mark.parametrize("tiling,kw", [
    ("block8n", dict(src=True)),
    ("ring", dict(src=True, ext_col=0)),
    ("persistent", dict(src=True, ext_col=-1)),
    ("strip12", dict(src=True)),
    ("block16", dict(integrator=bhr.BHR_RK4, ext_col=1)),
    ("block8", dict(precision=bhr.BHR_MIXED, src=True)),
    ("block8n", dict(precision=bhr.BHR_MIXED, ext_col=254)),
    ("block8n", dict(src=True, PTSX=800, PTSY=3000)),  # 38 MB a patch: sequences of one step
    ("block8n", dict(src=True, N=6400, M=64)),          # above the size that is captured
])
def test_any_split_of_a_run_gives_the_same_fields(tiling, kw, monkeypatch):
    monkeypatch.setenv("BHR_STAGE_TILING", tiling)
    kw = dict(kw)
    src, N, M = kw.pop("src", False), kw.pop("N", 256), kw.pop("M", 32)
    dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=200.0 * dt, Fr=3, out_start=0.0,
                     **{"ext_col": N * 6 // 10, **kw})
    if not src:
        prm.init_kind, prm.init_center = bhr.BHR_INIT_GAUSSIAN, 10.0 if prm.ext_col > 1 else -45.0
    rows = synthetic_plunge(prm.a, dt / 2.0, duration=prm.T)
    out = []
    for split in SPLITS:
        with bhr.Solver(prm) as s:
            assert s.info()["tiling"] == tiling
            if src:
                s.set_trajectory(rows)
            for n in split:
                s.step(n)
            out.append((s.get_state(), s.waveform(), s.psi_samples(), s.get_extraction(), s.get_source()))
    f0, w0, p0, e0, s0 = out[0]
    assert len(w0[0]) == 18 and np.max(np.abs(w0[1])) > 0
    for f, w, p, e, so in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(f0, f))
        assert np.array_equal(w0[0], w[0])
        assert np.linalg.norm(w[1] - w0[1]) <= 1e-13 * np.linalg.norm(w0[1])
        for a, b in zip(list(p0) + list(e0), list(p) + list(e)):
            assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(a)
        assert all(np.array_equal(a, b) for a, b in zip(s0, so))


@pytest.mark.parametrize("N,M,src", [(256, 32, True), (256, 32, False), (2048, 96, False), (6400, 64, True)])
def test_host_reads_see_a_single_steps_extraction(N, M, src):
    """A single step is extracted beside the next step, or by the first read
    that needs it: whatever is read after each of seven single steps (then a
    longer call, and single steps again) is what a run without reads has, on
    grids that run resident and by stage."""
    dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=100.0 * dt, Fr=2, out_start=0.0,
                     ext_col=N * 6 // 10, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=10.0)
    rows = synthetic_plunge(prm.a, dt / 2.0, duration=prm.T)
    readers = [lambda s: s.info()["rows_done"], lambda s: s.waveform(), lambda s: s.psi_samples(),
               lambda s: s.get_extraction(), lambda s: s.get_state(), lambda s: s.checkpoint(),
               lambda s: s.set_state(*s.get_state())]
    out = []
    for read in (True, False):
        with bhr.Solver(prm) as s:
            if src:
                s.set_trajectory(rows)
            for k in range(7):
                s.step(1)
                if read:
                    readers[k](s)
                    assert s.info()["rows_done"] == len(s.waveform()[0]) == k // 2 + 1
            for n in (20, 1, 1, 17, 1):
                s.step(n)
            assert s.info()["rows_done"] == 24
            out.append((s.get_state(), s.waveform(), s.psi_samples(), s.get_extraction()))
    (f0, w0, p0, e0), (f1, w1, p1, e1) = out
    assert all(np.array_equal(a, b) for a, b in zip(f0, f1)) and np.array_equal(w0[0], w1[0])
    for a, b in zip([w0[1], *p0, *e0], [w1[1], *p1, *e1]):
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)
