"""clbm_ref_perturbed_state at the largest sizes an int holds, where a count of
blocks rounded up by adding to n would overflow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2**31 - 1024, 2**31 - 512, 2**31 - 1])
def test_largest_states(gpu, clbm_lib, n):
    if gpu.cuda.mem_get_info()[0] < 4 * 8 * n:
        pytest.skip("needs 64 GB of free device memory")
    # f = c and one snapshot 2 c: the mix's weight is 1/2 (but for the last value,
    # 3e-10), so c becomes (c + eps c) / (1 + eps / 2); the norms' sums of n squares
    # leave a relative 1e-9 of room at most (n units of 2^-53)
    f = gpu.full((n,), 0.125, dtype=gpu.float64, device="cuda")
    snap = gpu.full((n,), 0.25, dtype=gpu.float64, device="cuda")
    f[-1] = 0.25  # the last value, on its own
    clbm_lib.ref_perturbed_state(f.data_ptr(), snap.data_ptr(), 0.5, 1, n, np.ones(1))
    lo, hi = float(f[:-1].min()), float(f[:-1].max())
    assert lo == hi and abs(hi - (0.125 + 0.5 * 0.125) / 1.25) < 1e-9
    assert abs(float(f[-1]) - (0.25 + 0.5 * 0.125) / 1.25) < 1e-9
    del f, snap
    gpu.cuda.empty_cache()
