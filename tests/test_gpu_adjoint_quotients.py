"""The FP64 adjoint's velocities are correctly rounded quotients.  A uniform flow
with jx = rho / 4 exactly has ux = 1/4 exactly, whatever the density; a product
with a rounded 1 / rho misses it for one density in five.  At the middle of the
square's upper side, under the momentum-exchange drag with tau = 1, no force and
one step, the collision's adjoint has exact operands up to a few roundings, so
the gradient's components along +y and -y are known to the bit (but for whether
the compiler fuses two of its products with the sums after them)."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, BOX = 12, 10, (4, 7, 3, 6)


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def components(rho):
    """the values that the +y and -y components may have"""
    ux, q, inv = 0.25, 4.0 * (1.0 / 36.0), 1.0 / rho
    gx, gy = rho * (3.0 * q), rho * (9.0 * (ux * -q))
    up, down = set(), set()
    for a in (3.0 * (ux * q) - (ux * gx) * inv, fma(-(ux * gx), inv, 3.0 * (ux * q))):
        up |= {a + gy * inv, fma(gy, inv, a)}
        down |= {a - gy * inv, fma(-gy, inv, a)}
    return up, down


def test_velocity_quotients(gpu, clbm_lib):
    rho = np.array([1.0 + (8 * j + 3) / 4096 if j % 2 else 1.0 - (8 * j + 5) / 8192 for j in range(256)])
    f = np.array([8, 5, 0.5, 1, 0.5, 0.25, 0.25, 0.25, 0.25]) / 16  # jx = rho / 4, jy = 0
    d = clbm_lib.RunDesc(width=W, height=H, xmin=BOX[0], xmax=BOX[1], ymin=BOX[2], ymax=BOX[3], nclones=len(rho),
                         ranks=1, tau=1.0, beta=0.0, alpha=0.0, force_scale=1.0, dt=1.0, drag_mode=1)
    with clbm_lib.Sampler([d], clbm_lib.FP64, max_steps=1) as s:
        s.load_run(0, (rho[:, None, None] * f).repeat(W * H, axis=1).ravel())
        s.drag_fwd(1, 1)
        s.drag_bwd()
        for j, r in enumerate(rho):
            g = s.drag_grad(0, j).reshape(W, H, 9)[5, BOX[3]]
            up, down = components(float(r))
            assert g[2] in up and g[4] in down, (j, r, g[2], up, g[4], down)
