"""clbm_get_run_variants and clbm_get_band_rows say what a run does: a run that was
given a cluster-resident variant but streams, because a row of an odd width takes
the room of one node more than the band has or because its square is one node
thick, reports the streaming variant and no bands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER2 = 8 + 3 + 1  # two bands, 512 threads


@pytest.mark.parametrize("W,H,thin,resident", [
    (97, 130, False, True),   # bands of 65 rows: 3185 pairs
    (97, 131, False, False),  # 66 rows: 3234 pairs of 3220
    (96, 132, False, True),   # 66 rows of an even width: 3168 pairs
    (20, 16, True, False),
])
def test_reported(gpu, clbm_lib, W, H, thin, resident):
    def desc(w, h, xmax):
        return clbm_lib.RunDesc(width=w, height=h, xmin=5, xmax=xmax, ymin=4, ymax=9, nclones=2, ranks=1, tau=0.57,
                                beta=2e-6, alpha=8.0, force_scale=100.0, dt=0.01)

    ds = [desc(W, H, 5 if thin else 9), desc(64, 24, 9)]
    out = []
    for variants in ([4, 4], [CLUSTER2, CLUSTER2]):
        with clbm_lib.Sampler(ds, clbm_lib.FP32, max_steps=12) as s:
            s.set_step_variant(4)
            s.set_run_variants(variants)
            got, bands = list(s.run_variants()), [len(s.band_rows(r)) for r in range(2)]
            if variants[0] != 4:
                assert got == [CLUSTER2 if resident else 4, CLUSTER2]
                assert bands == [2 if resident else 0, 2]
            s.set_run_variants(got)  # what was reported can be installed
            assert list(s.run_variants()) == got
            for r in range(2):
                s.init_equilibrium(r, 0.05, 1e-3, 7)
            s.run_interval(12)
            out.append([s.drag(r) for r in range(2)] + [s.dump(r, 1) for r in range(2)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
