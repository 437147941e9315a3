"""Whole steps of small source-free grids in one cooperative launch: each
tile stays on its SM, edges travel between neighbours stage by stage.

Against the oracle at the sizes where the tiling changes shape -- one strip
(both radial ends in one tile), one tile per column of strips, tiles of 3, 8,
9, 16, 17 and 32 rows (the limits of the kernel's three shapes on 148 SMs),
segments of uneven height, the first grid that does not fit -- with even and
odd m, the extraction column inside and at both ends, and step counts that
leave launches of 1, 63, 64 and a remainder.  Tolerances are those of the
other parity tests: fields 1e-12 of scale, waveform rows relative L2 1e-10,
times bit-identical."""
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


def test_a_trajectory_set_between_steps_leaves_the_resident_path():
    """Source-free steps (one launch), then sourced ones (by stage), against
    the oracle continued with the same state and a trajectory."""
    N, M, a = 512, 32, 0.6
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=a, m=2.0, dt=0.25 * 100.0 / N, T=60.0, Fr=5, out_start=0.0,
                     ext_col=320, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=5.0, init_width=2.0)
    rows = synthetic_plunge(a, prm.dt / 2.0, duration=prm.T)
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
