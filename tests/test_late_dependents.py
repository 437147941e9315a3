"""Stage launches of less than a wave of blocks let the next launch's blocks
in as their own end, larger ones at once.  Which it is changes when blocks
start, never what they read: at sizes on both sides of the rule's lines (148
SMs: up to 444 8-row tiles of four an SM, up to 296 16-row FP32 tiles of
three, and launches so small that two fit on different SMs) a run in one
sequence gives the same bits as single steps, whose final stage always lets
the extraction in at once, and agrees with 16-row tiles (two blocks an SM) to
1e-12 of scale (FP64; mixed 1e-6, the FP32 stages' rounding)."""
import numpy as np
import pytest

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.trajectory import synthetic_plunge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(512, 32), (1024, 64), (2048, 64), (3072, 64), (3520, 64), (3584, 64), (4096, 64),
                                 (4736, 64), (4800, 64)])
@pytest.mark.parametrize("kind", ["rk4", "mixed", "source"])
def test_fields_do_not_depend_on_when_blocks_start(N, M, kind, monkeypatch):
    dt = 0.25 * min(100.0 / N, 1.6 * np.pi / M)
    prm = bhr.Params(N=N, M=M, Xmin=-50.0, Xmax=50.0, a=0.6, m=2.0, dt=dt, T=100.0 * dt, Fr=3, out_start=0.0,
                     ext_col=N * 6 // 10, init_kind=bhr.BHR_INIT_GAUSSIAN, init_center=10.0,
                     integrator=bhr.BHR_RK4 if kind == "rk4" else bhr.BHR_SSPRK3,
                     precision=bhr.BHR_MIXED if kind == "mixed" else bhr.BHR_FP64)
    rows = synthetic_plunge(prm.a, dt / 2.0, duration=prm.T)
    out = []
    for tiling, split in (("block8n", [21]), ("block8n", [1] * 21), ("block16", [21])):
        monkeypatch.setenv("BHR_STAGE_TILING", tiling)
        with bhr.Solver(prm) as s:
            if kind == "source":
                s.set_trajectory(rows)
            for n in split:
                s.step(n)
            out.append(s.get_state())
    scale = max(np.max(np.abs(f)) for f in out[0])
    assert scale > 0 and all(np.array_equal(a, b) for a, b in zip(out[0], out[1]))
    tol = 1e-6 if kind == "mixed" else 1e-12
    assert max(np.max(np.abs(a - b)) for a, b in zip(out[0], out[2])) <= tol * scale
