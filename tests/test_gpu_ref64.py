"""The FP64 collision's shared divisor (csrc/clbm_physics.cuh) against the
oracle, bit for bit, on both sides of the rule that picks it: densities inside
and outside [0.5, 2), a density of all-ones significand, zero and tiny
momenta, no body force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,beta,kind", [
    (1.0, 1e-6, "noisy"), (1.0, 0.0, "noisy"), (0.5, 1e-6, "noisy"), (1.9999, 1e-6, "noisy"), (3.0, 1e-6, "noisy"),
    (0.3, 1e-6, "noisy"), (1e-200, 1e-6, "noisy"), (1.0, 1e-6, "rest"), (1.0, 1e-300, "rest"), (1.0, 1e-6, "ones"),
])
def test_stream_collide_equals_oracle(gpu, clbm_lib, orc, scale, beta, kind):
    torch = gpu
    g = orc.channel_geom(37, 19, 4, 9, 9)
    n = g.nx * g.ny
    rng = np.random.default_rng(11)
    if kind == "noisy":
        f = (orc.init_equilibrium(g, 0.05, 1e-2, 3, 0, 0).reshape(n, 9) * scale).copy()
    else:
        f = np.zeros((n, 9))
        f[:, 0] = 1.0 - 2.0 ** -53 if kind == "ones" else 1.0  # density of all-ones significand, or exactly 1
        if kind == "rest":
            f[::3, 1] = 2.0 ** -60 * rng.random(len(f[::3]))  # momenta far below the density's last place
            f[1::3, 2] = 1e-290
    f = np.ascontiguousarray(f.reshape(-1))
    want, fin, rho, ux, uy = orc.lbm_step(g, f, beta, 0.57)
    d = torch.from_numpy(f.copy()).cuda()
    out = torch.empty_like(d)
    macro = torch.empty(3, n, dtype=torch.float64, device="cuda")
    geom = clbm_lib.geom(g.nx, g.ny, g.xmin, g.xmax, g.ymin, g.ymax)
    clbm_lib.ref_stream_collide(geom, d.data_ptr(), out.data_ptr(), macro[0].data_ptr(), macro[1].data_ptr(),
                                macro[2].data_ptr(), beta, 0.57)
    torch.cuda.synchronize()
    # (the smallest densities overflow to infinities and NaN, at the same places)
    assert np.array_equal(d.cpu().numpy(), fin, equal_nan=True)
    assert np.array_equal(macro.cpu().numpy(), np.stack([rho, ux, uy]), equal_nan=True)
