"""The adjoint's forward through the cluster-resident kernel (checkpoints kept
as it steps) against the streaming steps: the drag integral,
the drag series and every gradient bit for bit, over checkpoint periods that
divide the interval, that do not, of one step and of more than the interval."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER_SIZES = (1, 2, 4, 8, 16, 3, 5, 6, 7, 9, 10)  # the variant numbering's order


@pytest.mark.parametrize("W,H,cs,tv,T,every", [
    (64, 24, 1, 1, 20, 5), (97, 33, 2, 1, 21, 8), (96, 23, 3, 2, 7, 1), (65, 40, 2, 0, 9, 30), (64, 24, 2, 1, 1, 3),
])
def test_resident_adjoint_equals_streaming(gpu, clbm_lib, W, H, cs, tv, T, every):
    nc, side = 3, 6
    xmin, ymin = W // 4 - side // 2, H // 2 - side // 2
    ds = [clbm_lib.RunDesc(width=W, height=H, xmin=xmin, xmax=xmin + side, ymin=ymin, ymax=ymin + side, nclones=nc,
                           ranks=1, tau=0.56, beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01, drag_mode=mode)
          for mode in (0, 1)]
    out = []
    for v in (4, 8 + 3 * CLUSTER_SIZES.index(cs) + tv):
        with clbm_lib.Sampler(ds, clbm_lib.FP32, max_steps=max(T, 2)) as s:
            s.set_step_variant(v)
            for r in range(2):
                s.init_equilibrium(r, 0.05, 1e-2, 9 + r)
            res = [s.drag_fwd(T, every)] + [s.drag(r) for r in range(2)]
            for _ in range(2):  # a backward pass may be repeated
                s.drag_bwd()
                res += [s.drag_grad(r, j) for r in range(2) for j in range(nc)]
            assert s.error_word() == 0
            out.append(res)
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
