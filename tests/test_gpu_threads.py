"""Contexts of different lattices stepping in threads of their own at the same time,
under the same kernel with different amounts of shared memory: no call is refused,
and every result is that of the context alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_intervals_in_threads(gpu, clbm_lib):
    lattices = [(256, 64, 4), (64, 40, 1), (120, 90, 2), (33, 150, 1)]  # width, height, cluster size
    rounds, T = 3000, 2

    def calls(W, H, cs, n):
        d = clbm_lib.RunDesc(width=W, height=H, xmin=8, xmax=14, ymin=9, ymax=15, nclones=2, ranks=1, tau=0.56,
                             beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01)
        out = []
        with clbm_lib.Sampler([d], clbm_lib.FP32, max_steps=T) as s:
            s.set_step_variant(8 + 3 * (1, 2, 4).index(cs) + 1)
            for _ in range(n):
                s.init_equilibrium(0, 0.05, 1e-3, 7)
                s.run_interval(T)
                out.append(s.drag(0))
        return out

    want = [calls(*lat, 1)[0] for lat in lattices]
    got = {}

    def work(i):
        try:
            got[i] = calls(*lattices[i], rounds)
        except clbm_lib.ClbmError as e:
            got[i] = e

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(lattices))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, res in got.items():
        assert isinstance(res, list), (lattices[i], res)
        for r in res:
            assert np.array_equal(r, want[i])
