"""FP64 steps and reseeds of a context of many runs: every run's results are those of
the run alone, bit for bit, and finding a block's run does not bound the step (a
step of a thousand runs of a clone takes no more than 2.5 times as long as one of a
run of a thousand clones; with the table of runs read one by one it took 6 times)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def desc(clbm_lib, r, W, H, nc, mode=0):
    return clbm_lib.RunDesc(width=W, height=H, xmin=W // 3, xmax=W // 3 + 4, ymin=H // 2 - 2, ymax=H // 2 + 2, nclones=nc,
                            ranks=1, tau=0.56, beta=2e-6, alpha=4.0, force_scale=100.0, dt=0.01, drag_mode=mode,
                            seed=r)


def test_many_runs_equal_each_alone(gpu, clbm_lib):
    T, lattices = 9, [(16 + 7 * (r % 5), 12 + 5 * (r % 4), 1 + r % 3, r % 2) for r in range(37)]
    # side 5 has 20 terms, a block of 64; a long one in the middle takes more
    ds = [desc(clbm_lib, r, *l) for r, l in enumerate(lattices)]
    ds[11] = clbm_lib.RunDesc(width=40, height=60, xmin=8, xmax=30, ymin=6, ymax=50, nclones=2, ranks=1, tau=0.56,
                              beta=2e-6, alpha=4.0, force_scale=100.0, dt=0.01, seed=11)

    def run(some):
        with clbm_lib.Sampler([ds[r] for r in some], clbm_lib.FP64, max_steps=T) as s:
            for i, r in enumerate(some):
                s.init_equilibrium(i, 0.05, 0.0, 0)
                rng = np.random.default_rng(r)
                for j in range(ds[r].nclones):
                    x = s.dump(i, j)
                    s.load(i, j, x * (1 + 1e-3 * rng.standard_normal(x.size)))
            s.run_interval(T)
            res = [s.drag(i) for i in range(len(some))]
            s.run_interval(T)  # the reseed's first collision, and again
            res = [[d, s.drag(i)] + [s.dump(i, j) for j in range(ds[r].nclones)]
                   for i, (d, r) in enumerate(zip(res, some))]
            assert s.error_word() == 0
            return res

    together = run(range(len(ds)))
    for r in range(len(ds)):
        for a, b in zip(together[r], run([r])[0]):
            assert np.isfinite(a).all() and np.array_equal(a, b), r


def test_finding_the_run(gpu, clbm_lib):
    T, ms = 40, []
    for nruns, nc in ((1, 1024), (1024, 1)):
        with clbm_lib.Sampler([desc(clbm_lib, r, 40, 24, nc) for r in range(nruns)], clbm_lib.FP64, max_steps=T) as s:
            for r in range(nruns):
                s.init_equilibrium(r, 0.05, 1e-3, 3)
            times = []
            for _ in range(5):
                s.profile(True)
                s.run_interval(T)
                s.sync()
                times.append(s.profile_read()[0])
            ms.append(min(times))
    assert ms[1] < 2.5 * ms[0], ms
