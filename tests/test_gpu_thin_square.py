"""Squares one node thick.  The cluster-resident kernel's in-place update needs
every slot to belong to one node, which such a square breaks, so a run with one
takes the streaming step under every variant: intervals, the adjoint and a batch
with an ordinary square beside it against the streaming variant, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER_SIZES = (1, 2, 4, 8, 16, 3, 5, 6, 7, 9, 10)  # the variant numbering's order
ORDINARY = (5, 9, 4, 9)


@pytest.mark.parametrize("box", [(5, 5, 5, 9), (5, 9, 5, 5), (5, 5, 5, 5)])
@pytest.mark.parametrize("cs,tv", [(1, 1), (2, 2), (3, 0), (None, None)])
def test_thin_square_streams(gpu, clbm_lib, box, cs, tv):
    nc, T = 3, 12

    def desc(b):
        return clbm_lib.RunDesc(width=20, height=16, xmin=b[0], xmax=b[1], ymin=b[2], ymax=b[3], nclones=nc, ranks=1,
                                tau=0.57, beta=2e-6, alpha=8.0, force_scale=100.0, dt=0.01,
                                perturb_mode=clbm_lib.PERTURB_UNIFORM, eps=1e-4, seed=7)

    def run(boxes, variant):
        with clbm_lib.Sampler([desc(b) for b in boxes], clbm_lib.FP32, max_steps=T) as s:
            if variant is None:  # as tuned, after an ordinary square on the same lattice has been
                with clbm_lib.Sampler([desc(ORDINARY) for _ in boxes], clbm_lib.FP32, max_steps=T) as o:
                    o.init_equilibrium(0, 0.05, 1e-3, 7)
                    o.autotune(2, measure=False)
                s.init_equilibrium(0, 0.05, 1e-3, 7)
                s.autotune(2, measure=False)
            else:
                s.set_step_variant(variant)
            res = []
            for r in range(len(boxes)):
                s.init_equilibrium(r, 0.05, 1e-3, 7 + r)
            res.append(s.drag_fwd(T, 5))
            s.drag_bwd()
            res += [s.drag_grad(r, j) for r in range(len(boxes)) for j in range(nc)]
            for steps in (T, T - 1, T):
                s.run_interval(steps)
                res += [s.drag(r) for r in range(len(boxes))]
                s.clone_step()
            s.run_interval(2)
            res += [s.dump(r, j) for r in range(len(boxes)) for j in range(nc)]
            assert s.error_word() == 0
            return res

    variant = None if cs is None else 8 + 3 * CLUSTER_SIZES.index(cs) + tv
    for boxes in ([box], [ORDINARY, box]):
        for got, want in zip(run(boxes, variant), run(boxes, 4)):
            assert np.isfinite(got).all() and np.array_equal(got, want)
