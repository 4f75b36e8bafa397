"""The pair kernel's last pair of a row of odd width has a lane without a node.  Its
values are nobody's, so the density test passes over them: in a channel that the
square blocks the flow stays slow, while an open column driven over as many steps
reaches speeds of a thousand and more, where FP32 no longer keeps its density."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cs,tv", [(1, 1), (2, 2)])
def test_blocked_channel(gpu, clbm_lib, cs, tv):
    W, H, T = 5, 400, 60000
    d = clbm_lib.RunDesc(width=W, height=H, xmin=0, xmax=W - 1, ymin=1, ymax=H - 2, nclones=1, ranks=1, tau=1.0,
                         beta=0.05, alpha=0.0, force_scale=1.0, dt=0.01)
    out = []
    for variant in (4, 8 + 3 * (1, 2).index(cs) + tv):
        with clbm_lib.Sampler([d], clbm_lib.FP32, max_steps=T) as s:
            s.set_step_variant(variant)
            assert list(s.run_variants()) == [variant]
            s.init_equilibrium(0, 0.0, 1e-3, 7)
            s.run_interval(T)
            assert s.error_word() == 0
            out.append((s.drag(0), s.dump(0, 0)))
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
