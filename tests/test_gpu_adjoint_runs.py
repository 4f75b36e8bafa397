"""The adjoint's forward with several cluster-resident runs in a context: the
runs step side by side, as in an interval (sixteen runs of a few clones, which
leave most of the chip idle, may take no more than six times one of them; one
after the other they take about sixteen times as long), and give the streaming
steps' integrals, drag series and gradients bit for bit."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T, EVERY, STREAM, CLUSTER3 = 100, 9, 4, 8 + 3 * 5 + 1  # variants: 128-node tiles, and 3 bands with 512 threads


def sampler(clbm_lib, nruns, variant, lattice=lambda r: (129, 129)):
    ds = []
    for r in range(nruns):
        W, H = lattice(r)
        ds.append(clbm_lib.RunDesc(width=W, height=H, xmin=W // 4, xmax=W // 4 + 8, ymin=H // 2 - 4, ymax=H // 2 + 4,
                                   nclones=2, ranks=1, tau=0.56, beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01))
    s = clbm_lib.Sampler(ds, clbm_lib.FP32, max_steps=T)
    s.set_step_variant(variant)
    for r in range(nruns):
        s.init_equilibrium(r, 0.05, 1e-2, 3 + r)
    return s


def test_runs_side_by_side(gpu, clbm_lib):
    ms = {}
    for nruns in (1, 16):
        with sampler(clbm_lib, nruns, CLUSTER3) as s:
            times = []
            for _ in range(6):  # the first allocates
                t = time.perf_counter()
                s.drag_fwd(T, EVERY)
                times.append(time.perf_counter() - t)
            ms[nruns] = min(times)
    assert ms[16] < 6 * ms[1], ms


def test_runs_equal_streaming(gpu, clbm_lib):
    nruns, out = 5, []
    for variant in (STREAM, CLUSTER3):
        with sampler(clbm_lib, nruns, variant, lambda r: (40 + 13 * r, 45 - 4 * r)) as s:
            res = []
            for every in (EVERY, 3):  # a forward pass may be repeated
                res.append(s.drag_fwd(T, every))
                res += [s.drag(r) for r in range(nruns)]
                s.drag_bwd()
                res += [s.drag_grad(r, j) for r in range(nruns) for j in range(2)]
            assert s.error_word() == 0
            out.append(res)
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
