"""Bands small enough for four CTAs an SM (784 pairs of nodes): with more blocks
than two an SM the 256-thread variant takes its kernel for them.  At that size, one
row above it, one-row bands, odd and the smallest widths, and with few clones, where
it does not: intervals and the adjoint against the streaming steps, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER_SIZES = (1, 2, 4, 8, 16, 3, 5, 6, 7, 9, 10)  # the variant numbering's order


@pytest.mark.parametrize("W,H,cs,nc", [
    (56, 28, 1, 400), (56, 29, 1, 400), (55, 28, 1, 400), (24, 16, 1, 3), (24, 16, 1, 1300), (3, 392, 1, 310),
    (5, 7, 2, 200), (50, 47, 3, 110), (1567, 4, 4, 80), (64, 24, 2, 160),
])
@pytest.mark.parametrize("field", [False, True])
def test_small_bands_equal_streaming(gpu, clbm_lib, W, H, cs, nc, field):
    if field and W > 1024:
        pytest.skip("no random field on this width")
    T, x0, y0 = 12, W // 4, max(1, H // 3)
    d = clbm_lib.RunDesc(width=W, height=H, xmin=x0, xmax=min(x0 + 5, W - 1), ymin=y0, ymax=min(y0 + 4, H - 2),
                         nclones=nc, ranks=1, tau=0.57, beta=2e-6, alpha=8.0, force_scale=100.0, dt=0.01,
                         perturb_mode=clbm_lib.PERTURB_UNIFORM, eps=1e-4, seed=7)
    if field:
        d.field_mode, d.field_steps, d.field_eps, d.field_sigma = 1, 7, 0.2, 6.0
    some, out = sorted({0, 1, nc // 2, nc - 1}), []
    for variant in (4, 8 + 3 * CLUSTER_SIZES.index(cs) + 2):
        with clbm_lib.Sampler([d], clbm_lib.FP32, max_steps=T) as s:
            s.set_step_variant(variant)
            assert list(s.run_variants()) == [variant]
            s.init_equilibrium(0, 0.05, 1e-3, 7)
            res = []
            for steps in (T, T - 1):
                s.run_interval(steps)
                res.append(s.drag(0))
                s.clone_step()
            s.run_interval(T)
            if not field:
                res.append(s.drag_fwd(T, 5))
                s.drag_bwd()
                res += [s.drag_grad(0, j) for j in some]
            res += [s.dump(0, j) for j in some]
            assert s.error_word() == 0
            out.append(res)
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
