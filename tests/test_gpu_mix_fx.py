"""The snapshot mix's fixed-point sums (csrc/clbm_refops.cu): the perturbation
that keeps the mix of its first pass and the one that forms it again in FP64
must give the same bits, on both sides of the rule on the prefactors, with
values of every size in the snapshots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsnap", [1, 2, 3, 10, 33, 64])
@pytest.mark.parametrize("pre", ["random", "small_first", "tiny_first", "zeros", "negative", "large", "minute"])
@pytest.mark.parametrize("kind", ["states", "any"])
def test_kept_mix_equals_fp64_mix(gpu, clbm_lib, nsnap, pre, kind):
    torch = gpu
    rng = np.random.default_rng(nsnap)
    n = 9 * 331
    w = np.tile(np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4), n // 9)
    if kind == "states":
        f, snaps = (w * (1 + 0.1 * rng.uniform(-1, 1, (1, n))) for _ in range(2))
        snaps = w * (1 + 0.1 * rng.uniform(-1, 1, (nsnap, n)))
    else:  # exponents of their own, zeros, short significands, a few negative values
        f = w[None, :].copy()
        snaps = 2.0 ** rng.uniform(-60, 2, (nsnap, n)) * rng.choice([1.0, 1.0, 1.0, 0.0, -1.0], (nsnap, n))
        snaps = np.where(rng.random((nsnap, n)) < 0.5, w * rng.integers(1, 9, (nsnap, n)) / 8, snaps)
    r = rng.random(nsnap)
    if pre == "small_first":
        r[0] = 0.05
    elif pre == "tiny_first":
        r[0] = 1e-9
    elif pre == "zeros":
        r[1:] = 0.0
    elif pre == "negative":
        r[-1] = -r[-1]
    elif pre == "large":
        r *= 1e5
    elif pre == "minute":
        r *= 1e-5
    d_snaps = torch.from_numpy(np.ascontiguousarray(snaps)).cuda()
    out = []
    for call in (clbm_lib.ref_perturbed_state, clbm_lib.ref_perturbed_state_noalloc):
        d = torch.from_numpy(f.reshape(-1).copy()).cuda()
        call(d.data_ptr(), d_snaps.data_ptr(), 0.7, nsnap, n, np.ascontiguousarray(r))
        torch.cuda.synchronize()
        out.append(d.cpu().numpy())
    assert np.array_equal(out[0], out[1], equal_nan=True)
