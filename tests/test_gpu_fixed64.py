"""The FP64 collision's fixed-point sums (csrc/clbm_physics.cuh) against the
oracle, bit for bit, on both sides of the rules that pick them: speeds about
0.148, populations about 2^-9, 2^-7 and 1/4, sums that cancel, relaxation
times at which the old populations count nothing, all or more, drives from
nothing to larger than the populations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CX = np.array([0, 1, 0, -1, 0, 1, -1, -1, 1])
CY = np.array([0, 0, 1, 0, -1, 1, 1, -1, -1])
W = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)


def _state(kind, n, rng):
    warp = np.arange(n) // 32
    if kind == "speed":  # warps slower than the limit, faster, and of both
        lim = np.where(warp % 3 == 0, 0.13, np.where(warp % 3 == 1, 0.148, 0.2))
        ux, uy = rng.uniform(-1, 1, (2, n)) * lim
        eu = CX * ux[:, None] + CY * uy[:, None]
        f = W * (1 + 3 * eu + 4.5 * eu**2 - 1.5 * (ux**2 + uy**2)[:, None])
        return f * (1 + 1e-3 * rng.uniform(-1, 1, f.shape))
    if kind == "edges":  # neighbours of the powers of two that bound the ranges
        f = W * (1 + 1e-2 * rng.uniform(-1, 1, (n, 9)))
        at = rng.random((n, 9)) < 0.1
        at[:, 0] = False
        edge = rng.choice([2.0**-9, 2.0**-8, 2.0**-7, 0.25], (n, 9)) * rng.choice([1 - 2.0**-53, 1, 1 + 2.0**-52], (n, 9))
        return np.where(at & (warp % 2 == 0)[:, None], edge, f)
    # any exponent, in every third warp of both signs
    f = 2.0 ** rng.uniform(-11, -1, (n, 9))
    f[:, 0] += 0.2
    return np.where((rng.random((n, 9)) < 0.2) & (warp % 3 == 0)[:, None] & (CX != 0), -f, f)


@pytest.mark.parametrize("tau", [0.5000001, 0.56, 0.99, 1.0, 1.0 + 2.0**-40, 7.0])
@pytest.mark.parametrize("kind,beta", [("speed", 1e-6), ("speed", 0.0), ("edges", 1e-5), ("edges", 1e-18),
                                       ("any", 1e-6), ("any", 0.4), ("speed", 1.2)])
def test_stream_collide_equals_oracle(gpu, clbm_lib, orc, kind, beta, tau):
    torch = gpu
    g = orc.channel_geom(53, 31, 4, 9, 9)
    n = g.nx * g.ny
    f = np.ascontiguousarray(_state(kind, n, np.random.default_rng(5)).reshape(-1))
    want, fin, rho, ux, uy = orc.lbm_step(g, f, beta, tau)
    d = torch.from_numpy(f.copy()).cuda()
    out = torch.empty_like(d)
    macro = torch.empty(3, n, dtype=torch.float64, device="cuda")
    geom = clbm_lib.geom(g.nx, g.ny, g.xmin, g.xmax, g.ymin, g.ymax)
    clbm_lib.ref_stream_collide(geom, d.data_ptr(), out.data_ptr(), macro[0].data_ptr(), macro[1].data_ptr(),
                                macro[2].data_ptr(), beta, tau)
    torch.cuda.synchronize()
    assert np.array_equal(macro.cpu().numpy(), np.stack([rho, ux, uy]), equal_nan=True)
    assert np.array_equal(d.cpu().numpy(), fin, equal_nan=True)
