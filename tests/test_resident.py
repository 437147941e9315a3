"""Whole steps of small grids in one cooperative launch: each tile stays on
its SM, edges travel between neighbours stage by stage.

Against the oracle at the sizes where the tiling changes shape -- one strip
(both radial ends in one tile), one tile per column of strips, tiles of 3, 8,
9, 16, 17 and 32 rows (the limits of the kernel's three shapes on 148 SMs),
segments of uneven height, the first grid that does not fit -- with even and
odd m, the extraction column inside and at both ends, and step counts that
leave launches of 1, 63, 64 and a remainder.  With a source and with RK4
against the stage launches.  Tolerances are those of the other parity tests:
fields 1e-12 of scale, waveform rows relative L2 1e-10, times bit-identical."""
import threading

import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge
from oracle import pyoracle

pytestmark = pytest.mark.gpu

FIELD_TOL, WAVE_TOL = 1e-12, 1e-10


def params(N, M, m, ext_col, T=50.0, Fr=5):
    centre = 0.0 if 2 < ext_col < N - 3 else (12.0 if ext_col > 2 or ext_col < 0 else -15.0)
    return bhr.Params(N=N, M=M, Xmin=-20.0, Xmax=20.0, a=0.7, m=float(m), dt=0.2 * min(40.0 / N, 1.7 * np.pi / M), T=T,
                      Fr=Fr, out_start=0.0, ext_col=ext_col, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=centre,
                      init_width=2.0, init_ell=float(max(2, abs(m))))


def field_err(got, want):
    scale = max(np.max(np.abs(w)) for w in want)
    return max(np.max(np.abs(g - w)) for g, w in zip(got, want)) / scale


@pytest.mark.parametrize("N,M,m,ext_col", [
    (64, 16, 2, 30),      # one strip, 3-row tiles
    (64, 512, 2, 40),     # one strip, every SM a segment
    (256, 32, -3, 0),     # extraction at the inner end
    (896, 80, 1, 1),      # 8-row tiles, an inner closure column
    (1024, 80, 2, -1),    # 9-row tiles (two columns a thread), the outer end
    (1984, 64, 3, 1200),  # 15-row tiles, segments of uneven height
    (1152, 128, -2, 700),  # 16-row tiles
    (896, 176, 2, 894),   # 17-row tiles (two rows a warp), an outer closure column
    (1152, 256, -1, 500),  # 32-row tiles
    (9472, 32, 2, 4700),  # 148 strips, one segment of 26 rows
])
def test_small_grids_match_the_oracle(N, M, m, ext_col):
    prm = params(N, M, m, ext_col)
    with bhr.Solver(prm) as s:
        assert s.info()["tiling"] == "resident", s.info()
        for n in (1, 63, 66):
            s.step(n)
        got, (t, h, e), ext, samples = s.get_state(), s.waveform(), s.get_extraction(), s.psi_samples()
        assert s.info()["steps_done"] == 130
    o = pyoracle.Oracle(N, M, prm.Xmin, prm.Xmax, prm.a, prm.m, prm.dt, T=prm.T, Fr=5, out_start=0.0, ext_col=ext_col)
    o.init_gaussian(prm.init_center, prm.init_width, prm.init_ell)
    ot, oh, oe, *_ = o.run(nsteps=130)
    assert field_err(got, o.get_state()) <= FIELD_TOL
    assert len(t) == 26 and np.array_equal(t, ot)
    assert np.linalg.norm(h - oh) <= WAVE_TOL * np.linalg.norm(oh)
    assert np.linalg.norm(e - oe) <= WAVE_TOL * np.linalg.norm(oe)
    er, ei = o.ext()
    assert np.linalg.norm(np.concatenate([ext[0] - er, ext[1] - ei])) <= WAVE_TOL * np.linalg.norm(er)
    assert samples[0].shape == (26, M)


def test_grids_that_do_not_fit_run_by_stage():
    for N, M in ((9536, 16), (4096, 80)):  # more strips than SMs; tiles of 37 rows
        with bhr.Solver(params(N, M, 2, N // 2)) as s:
            assert s.info()["tiling"] != "resident"


@pytest.mark.parametrize("N,M,src,rk4,kw", [
    (64, 16, True, True, {}),       # 3-row tiles, one strip
    (512, 32, True, False, {}),     # 3-row tiles
    (896, 80, True, True, {}),      # 8-row tiles
    (1024, 80, True, False, {}),    # 9-row tiles (two columns a thread)
    (1024, 80, False, True, {}),
    (1152, 128, True, False, {}),   # 16-row tiles, the tallest with a source and of RK4
    (1152, 128, True, True, {}),
    (9472, 16, False, True, {}),    # 148 strips
    (512, 32, True, False, dict(PTSX=800, PTSY=3000)),  # two patch buffers: two steps a launch
])
def test_source_and_rk4_match_the_steps_by_stage(N, M, src, rk4, kw):
    """A trajectory and RK4's four stages against the stage launches (which
    the other parity tests hold to the oracle): a trajectory set after 70
    steps, then launches of 1, 64 and fewer steps."""
    T, dt = 60.0, 0.25 * min(100.0 / N, 1.5 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=T, Fr=5, out_start=0.0, ext_col=N * 5 // 8,
                     integrator=bhr.BHR_RK4 if rk4 else bhr.BHR_SSPRK3, init_kind=bhr.BHR_INIT_GAUSSIAN,
                     init_center=5.0, init_width=2.0, **kw)
    rows = synthetic_plunge(prm.a, dt / 2.0, duration=T)
    out, saved = [], None
    for tiling in (None, "block8n", None):  # the third resumes the second's checkpoint
        with pytest.MonkeyPatch.context() as mp:
            if tiling:
                mp.setenv("BHR_STAGE_TILING", tiling)
            with bhr.Solver(prm) as s:
                if len(out) < 2:
                    s.step(70)
                if src:
                    s.set_trajectory(rows)
                assert (s.info()["tiling"] == "resident") == (tiling is None)
                if len(out) < 2:
                    s.step(1)
                    saved = s.checkpoint()
                else:
                    s.restore(saved)
                for n in (66, 3):
                    s.step(n)
                out.append((s.get_state(), s.waveform(), s.get_extraction(), s.get_source()))
    f1, w1, e1, s1 = out[1]
    for f, w, e, so in (out[0], out[2]):
        assert field_err(f, f1) <= FIELD_TOL and np.array_equal(w[0], w1[0])
        assert np.linalg.norm(w[1] - w1[1]) <= WAVE_TOL * np.linalg.norm(w1[1])
        assert np.linalg.norm(e[0] - e1[0]) <= WAVE_TOL * np.linalg.norm(e1[0])
        assert all(np.array_equal(x, y) for x, y in zip(so, s1)) and (not src or np.max(np.abs(s1[0])) > 0)


def test_a_source_on_taller_tiles_leaves_the_resident_path():
    """Source-free steps (one launch), then sourced ones (by stage) on a grid
    of 19-row tiles, against all steps by stage."""
    prm = bhr.Params(N=2048, M=80, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=0.012, T=3.0, Fr=5, out_start=0.0,
                     ext_col=1280, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=5.0, init_width=2.0)
    rows = synthetic_plunge(prm.a, prm.dt / 2.0, duration=prm.T)
    out = []
    for tiling in (None, "block8n"):
        with pytest.MonkeyPatch.context() as mp:
            if tiling:
                mp.setenv("BHR_STAGE_TILING", tiling)
            with bhr.Solver(prm) as s:
                s.step(70)
                assert (s.info()["tiling"] == "resident") == (tiling is None)
                s.set_trajectory(rows)
                assert s.info()["tiling"] != "resident"
                s.step(60)
                out.append((s.get_state(), s.waveform()))
    (f0, w0), (f1, w1) = out
    assert field_err(f0, f1) <= FIELD_TOL and np.array_equal(w0[0], w1[0])
    assert np.linalg.norm(w0[1] - w1[1]) <= WAVE_TOL * np.linalg.norm(w1[1])


def test_solves_on_several_threads_do_not_disturb_each_other():
    """Each of four solves (other grids, spins and m) stepped on its own
    thread gives the bits it gives alone."""
    prms = [params(1024, 64, 2, 600), params(1216, 80, -3, -1), params(2048, 64, 1, 900), params(256, 32, 2, 130)]

    def run(prm, out, i):
        with bhr.Solver(prm) as s:
            for _ in range(12):
                s.step(17)
            out[i] = (s.get_state(), s.waveform())

    alone, together = [None] * 4, [None] * 4
    for i, prm in enumerate(prms):
        run(prm, alone, i)
    threads = [threading.Thread(target=run, args=(prm, together, i)) for i, prm in enumerate(prms)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for (fa, wa), (ft, wt) in zip(alone, together):
        assert all(np.array_equal(x, y) for x, y in zip(fa, ft))
        assert all(np.array_equal(x, y) for x, y in zip(wa, wt))


@pytest.mark.parametrize("N,M,m", [(64, 16, 2), (256, 32, -1), (1216, 96, 3), (64, 1024, 2)])
def test_noalloc_closes_the_state_it_leaves(N, M, m):
    """The state in the caller's memory after a resident call, boundary rows
    and columns included, against the oracle's; then another grid (its edge
    words laid out differently) and the first again, on the same scratch."""
    import torch

    def go(prm, steps):
        o = pyoracle.Oracle(prm.N, prm.M, prm.Xmin, prm.Xmax, prm.a, prm.m, prm.dt, T=prm.T, Fr=5, out_start=0.0)
        o.init_gaussian(prm.init_center, prm.init_width, prm.init_ell)
        state = torch.from_numpy(np.stack(o.get_state())).to("cuda")
        torch.cuda.synchronize()
        for n in steps:
            bhr.step_noalloc(prm, state.data_ptr(), n)
            o.step(n)
        return field_err(state.cpu().numpy(), o.get_state())

    small, wide = params(N, M, m, 30), params(8192, 16, 2, 4000)
    assert go(small, (1, 0, 9)) <= FIELD_TOL
    assert go(wide, (3,)) <= FIELD_TOL
    assert go(small, (5,)) <= FIELD_TOL
