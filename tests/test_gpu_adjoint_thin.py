"""The adjoint of a run whose square is one node thick: there a post-collision
population may be read by two slots (the node's own, bounced back, and a
neighbour's), or by none.  Both precisions against central differences of the
FP64 forward, at the tolerances of the ordinary squares' test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(12, 12, 9, 14), (9, 14, 12, 12), (12, 12, 12, 12), (0, 0, 1, 22), (3, 9, 1, 1)])
def test_thin_square_adjoint(gpu, clbm_lib, box):
    nc, T, every, eps, (W, H) = 2, 20, 7, 1e-6, (32, 24)
    d = clbm_lib.RunDesc(width=W, height=H, xmin=box[0], xmax=box[1], ymin=box[2], ymax=box[3], nclones=nc, ranks=1,
                         tau=0.6, beta=1e-5, alpha=1.0, force_scale=100.0, force_shift=0.0, dt=0.01)
    n = 9 * W * H
    rng = np.random.default_rng(5)
    w = np.tile(np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4), nc * W * H)
    S0 = w * (1 + 1e-2 * rng.uniform(-1, 1, w.size))
    grad = {}
    for prec in (clbm_lib.FP64, clbm_lib.FP32):
        with clbm_lib.Sampler([d], prec, max_steps=T) as s:
            s.load_run(0, S0)
            s.drag_fwd(T, every)
            s.drag_bwd()
            grad[prec] = np.concatenate([s.drag_grad(0, j) for j in range(nc)]).reshape(nc, n)
    gnorm = np.linalg.norm(grad[clbm_lib.FP64], axis=1)
    # (the drag of a single node is zero, and so is its gradient)
    assert ((gnorm > 0) == (box[0] != box[1] or box[2] != box[3])).all()
    assert (np.linalg.norm(grad[clbm_lib.FP32] - grad[clbm_lib.FP64], axis=1) <= 1e-5 * gnorm).all()
    with clbm_lib.Sampler([d], clbm_lib.FP64, max_steps=T) as f:
        for _ in range(4):
            dirn = rng.normal(0.0, 1.0, S0.size)
            f.load_run(0, S0 + eps * dirn)
            jp = f.drag_fwd(T, every)
            f.load_run(0, S0 - eps * dirn)
            jm = f.drag_fwd(T, every)
            fd = (jp - jm) / (2 * eps)
            dn = np.linalg.norm(dirn.reshape(nc, n), axis=1)
            for prec, tol in ((clbm_lib.FP64, 1e-10), (clbm_lib.FP32, 1e-6)):
                ad = (grad[prec] * dirn.reshape(nc, n)).sum(axis=1)
                assert (np.abs(ad - fd) <= tol * gnorm * dn).all(), (prec, ad, fd)
