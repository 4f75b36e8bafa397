"""clbm_ref_perturbed_state and its variant without allocation on both sides of the
size up to which the norms take one value per thread (77824), and of a block: the
same bits from both, and the extended-precision result within what the operations'
roundings leave: nsnap + 2 in a mix, under 100 in the chains of the norms' sums and
the update, half a unit of 2^-52 each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 9 * 12 * 9, 77823, 77824, 77825, 9 * 97 * 97])
@pytest.mark.parametrize("nsnap", [1, 2, 10, 40])
@pytest.mark.parametrize("first", [0.6, -0.6])
def test_sizes(gpu, clbm_lib, n, nsnap, first):
    rng = np.random.default_rng(n + nsnap)
    w = np.resize(np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4), n)
    f = w * (1 + 0.1 * rng.uniform(-1, 1, n))
    snaps = w * (1 + 0.1 * rng.uniform(-1, 1, (nsnap, n)))
    pre = rng.uniform(0.2, 1.0, nsnap)
    pre[0] = first
    if first < 0 and nsnap == 2:
        pre[1] = 1.5  # (away from a mix of nothing)
    d_snaps = gpu.from_numpy(snaps.reshape(-1)).cuda()
    out = []
    for call in (clbm_lib.ref_perturbed_state, clbm_lib.ref_perturbed_state_noalloc):
        d = gpu.from_numpy(f.copy()).cuda()
        call(d.data_ptr(), d_snaps.data_ptr(), 0.05, nsnap, n, pre)
        out.append(d.cpu().numpy())
    assert np.array_equal(*out)
    wide = np.longdouble
    mix, size = np.zeros(n, wide), np.zeros(n, wide)
    for p, s in zip(pre, snaps):
        mix += wide(p) * s.astype(wide)
        size += abs(wide(p)) * s.astype(wide)
    weight = np.sqrt((f.astype(wide) ** 2).sum()) / np.sqrt((mix ** 2).sum())
    a = 1 + wide(pre.sum()) * wide(0.05) * weight
    want = (f.astype(wide) + wide(0.05) * mix * weight) / a
    scale = (abs(f) + wide(0.05) * size * weight) / abs(a)
    assert (abs(out[0] - want) <= (nsnap + 102) * wide(2) ** -53 * scale * (1 + abs(size / mix).max())).all()
