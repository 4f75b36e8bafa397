"""The cluster-resident interval kernel takes two nodes of a row per thread
(x and x + ceil(W/2)); its row ends, empty lane (odd widths), walls, band edges
and the square's perimeter against the streaming step kernel, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER_SIZES = (1, 2, 4, 8, 16, 3, 5, 6, 7, 9, 10)  # the variant numbering's order


def variant(cs, tv):
    return 8 + 3 * CLUSTER_SIZES.index(cs) + tv


@pytest.mark.parametrize("W,H,xmin,xmax,ymin,ymax,cs,tv,rows,field", [
    (97, 33, 21, 27, 13, 19, 2, 1, None, False),       # odd width
    (129, 41, 50, 80, 18, 24, 3, 0, [19, 3, 19], False),  # odd width, square over both halves and two band edges
    (65, 40, 0, 12, 10, 22, 3, 2, None, True),         # square at the periodic wrap
    (66, 24, 53, 65, 8, 16, 2, 1, None, False),        # ... at the other end
    (33, 17, 13, 20, 6, 10, 1, 1, None, False),
    (11, 13, 4, 7, 4, 7, 2, 2, None, True),            # rows shorter than a warp
    (3, 50, 0, 1, 20, 24, 1, 0, None, False),          # two pairs per row
    (130, 26, 30, 36, 11, 15, 4, 1, [1, 12, 12, 1], False),  # one-row bands
    (64, 12, 20, 44, 1, 10, 3, 1, None, False),        # square next to both walls, in every band
    (130, 60, 40, 52, 24, 36, 2, 2, None, True),       # 256 threads with planes of the full size
    (97, 66, 20, 33, 25, 38, 1, 1, None, False),       # accepted, but one node per row too large: streams
])
def test_pairs_equal_streaming(gpu, clbm_lib, W, H, xmin, xmax, ymin, ymax, cs, tv, rows, field):
    u0, nc, T = 0.05, 3, 11
    d = clbm_lib.RunDesc(width=W, height=H, xmin=xmin, xmax=xmax, ymin=ymin, ymax=ymax, nclones=nc, ranks=1, tau=0.57,
                         beta=2e-6, alpha=8.0, force_scale=100.0, dt=0.01, perturb_mode=clbm_lib.PERTURB_UNIFORM,
                         eps=1e-4, seed=7)
    if field:
        d.field_mode, d.field_steps, d.field_eps, d.field_sigma = 1, 5, 0.2, 6.0
    out = []
    for v in (4, variant(cs, tv)):
        with clbm_lib.Sampler([d], clbm_lib.FP32, max_steps=T) as s:
            s.set_step_variant(v)
            if rows and v != 4:
                s.set_band_rows(0, rows)
            s.init_equilibrium(0, u0, 1e-3, 7)
            res = []
            for steps in (T, T - 1, 1, 2):  # last steps of both kinds, with and without the reseed in the load
                s.run_interval(steps)
                res.append(s.drag(0))
                s.clone_step()
                res.append(s.clone_result(0)["labels"])
            s.run_interval(T)
            res += [s.drag(0)] + [s.dump(0, j) for j in range(nc)]
            assert s.error_word() == 0
            out.append(res)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
