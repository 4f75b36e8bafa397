"""clbm_ref_perturbed_state where the device has no room for the state's mix
beside the state and its snapshots: the mix is formed twice instead of kept, the
same result bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_without_room_for_the_mix(gpu, clbm_lib):
    n, nsnap, eps, pre = 1 << 29, 2, 0.05, np.array([0.6, 0.3])  # the mix: 4 GB
    gpu.cuda.empty_cache()
    g = gpu.Generator(device="cuda").manual_seed(11)
    snaps = gpu.empty(nsnap * n, dtype=gpu.float64, device="cuda").uniform_(0.1, 0.12, generator=g)
    out = []
    for room in (True, False):
        f = gpu.empty(n, dtype=gpu.float64, device="cuda").uniform_(0.1, 0.12, generator=g.manual_seed(12))
        gpu.cuda.synchronize()
        held = None if room else gpu.empty(gpu.cuda.mem_get_info()[0] - (2 << 30), dtype=gpu.uint8, device="cuda")
        clbm_lib.ref_perturbed_state(f.data_ptr(), snaps.data_ptr(), eps, nsnap, n, pre)
        del held
        gpu.cuda.empty_cache()
        out.append(f)
    assert gpu.equal(*out)
