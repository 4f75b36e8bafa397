"""The FP64 step of a context with one run takes the run from its launch
parameters and reads the table of runs otherwise: a context of two runs must
give each what a context of its own gives it, bit for bit, both drags.
Perimeters of fewer drag terms than a block has threads, of as many, one more
and several blocks of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# W, H, square, clones, drag mode; drag terms 28, 64 (a block), 66, 146
RUNS = [(48, 30, (10, 16, 9, 15), 3, 0), (41, 37, (8, 23, 9, 24), 2, 1), (64, 40, (9, 25, 10, 25), 2, 0),
        (96, 64, (20, 55, 12, 48), 1, 1)]


def desc(lib, W, H, sq, nc, mode):
    return lib.RunDesc(width=W, height=H, xmin=sq[0], xmax=sq[1], ymin=sq[2], ymax=sq[3], nclones=nc, ranks=1,
                       tau=0.57, beta=1e-5, alpha=3.0, force_scale=10.0, dt=0.01,
                       perturb_mode=lib.PERTURB_UNIFORM, eps=1e-4, seed=9, drag_mode=mode)


@pytest.mark.parametrize("i,j", [(0, 1), (1, 2), (2, 3), (3, 0)])
def test_two_runs_equal_each_alone(gpu, clbm_lib, i, j):
    T, rng = 7, np.random.default_rng(4)
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    runs = [RUNS[i], RUNS[j]]
    states = [[(w * (1 + 0.05 * rng.uniform(-1, 1, (r[0] * r[1], 9)))).reshape(-1) for _ in range(r[3])] for r in runs]

    def go(which):
        with clbm_lib.Sampler([desc(clbm_lib, *runs[q]) for q in which], clbm_lib.FP64, max_steps=T) as s:
            for p, q in enumerate(which):
                for c, f in enumerate(states[q]):
                    s.load(p, c, f)
            s.run_interval(T)
            return [(s.drag(p), [s.dump(p, c) for c in range(runs[q][3])]) for p, q in enumerate(which)]

    both = go([0, 1])
    for q in (0, 1):
        drag, pops = go([q])[0]
        assert np.array_equal(both[q][0], drag)
        for a, b in zip(both[q][1], pops):
            assert np.array_equal(a, b)
