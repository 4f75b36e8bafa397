"""A launch that the CUDA runtime refuses (the drag of a square whose terms do not
fit a block's shared memory) is an error of that call alone: the calls after it,
this library's and torch's, work as before."""
import pytest

pytestmark = pytest.mark.gpu


def test_next_call_works(gpu, clbm_lib):
    n, side = 1700, 1600  # 4 (side + 1) terms of 8 bytes, above 48 KB
    g = clbm_lib.geom(n, n, 40, 40 + side, 40, 40 + side)
    f = gpu.ones(9 * n * n, dtype=gpu.float64, device="cuda")
    d = clbm_lib.RunDesc(width=40, height=24, xmin=8, xmax=14, ymin=9, ymax=15, nclones=2, ranks=1, tau=0.56,
                         beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01)
    for prec in (clbm_lib.FP32, clbm_lib.FP64):
        with clbm_lib.Sampler([d], prec, max_steps=4) as s:
            s.init_equilibrium(0, 0.05, 1e-3, 7)
            with pytest.raises(clbm_lib.ClbmError):
                clbm_lib.ref_force_on_square(g, f.data_ptr(), 1.7)
            s.run_interval(4)
            s.sync()
            assert s.error_word() == 0
            with pytest.raises(clbm_lib.ClbmError):
                clbm_lib.ref_force_on_square(g, f.data_ptr(), 1.7)
            s.clone_step()
            assert s.drag(0).shape[0] == 2
    with pytest.raises(clbm_lib.ClbmError):
        clbm_lib.ref_force_on_square(g, f.data_ptr(), 1.7)
    assert float((f[:10] + 1).sum()) == 20.0
