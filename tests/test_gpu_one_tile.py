"""FP32 streaming step on lattices that fit one tile of a launch shape (128, 256
or 512 nodes): with several clones in one context, every streaming variant gives
each clone what a context of that clone alone gives, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(7, 9), (16, 8), (13, 10), (16, 16), (20, 15), (32, 16), (27, 19)])
def test_clones_of_one_tile(gpu, clbm_lib, W, H):
    nc, T = 3, 6

    def desc(n):
        return clbm_lib.RunDesc(width=W, height=H, xmin=2, xmax=4, ymin=3, ymax=5, nclones=n, ranks=1, tau=0.6,
                                beta=1e-5, alpha=1.0, force_scale=100.0, dt=0.01)

    rng = np.random.default_rng(W * H)
    w = np.tile(np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4), W * H)
    states = w * (1 + 1e-2 * rng.standard_normal((nc, w.size)))

    def run(some, variant):
        with clbm_lib.Sampler([desc(len(some))], clbm_lib.FP32, max_steps=T) as s:
            s.set_step_variant(variant)
            for j, f in enumerate(some):
                s.load(0, j, f)
            s.run_interval(T)
            assert s.error_word() == 0
            return [(s.drag(0)[j], s.dump(0, j)) for j in range(len(some))]

    alone = [run(states[j:j + 1], 0)[0] for j in range(nc)]
    for variant in range(8):
        for got, want in zip(run(states, variant), alone):
            assert np.isfinite(got[0]).all() and np.array_equal(got[0], want[0]), variant
            assert np.array_equal(got[1], want[1]), variant
