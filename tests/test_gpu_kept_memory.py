"""The device memory that the library keeps between calls: given back by
clbm_destroy(NULL) and with the last context, and shared by threads with streams
of their own without a change of any result."""
import os
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PKG = Path(__file__).resolve().parent.parent / "cloning-lbm-mpi_gb300"

GIVEN_BACK = """
import numpy as np, torch, clbm

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

L, n = clbm.lib(), 3 << 20
f = torch.full((n,), 0.1, dtype=torch.float64, device="cuda")
snap = f.clone()

def perturb(n):
    clbm.ref_perturbed_state(f.data_ptr(), snap.data_ptr(), 0.05, 1, n, np.ones(1))

def context():
    d = clbm.RunDesc(width=600, height=400, xmin=20, xmax=40, ymin=90, ymax=110, nclones=1, ranks=1, tau=0.56,
                     beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01)
    with clbm.Sampler([d], clbm.FP64, max_steps=2) as s:
        s.init_equilibrium(0, 0.05, 1e-3, 7)
        s.run_interval(2)
        s.dump(0, 0)

perturb(900), context()  # modules loaded, the pool made
L.clbm_destroy(None)
start = free()
perturb(n)
kept = start - free()
assert 8 * n <= kept <= 64 << 20, kept
assert L.clbm_destroy(None) == 0
assert free() == start, (free(), start)
perturb(n)
context()
assert free() == start, (free(), start)
"""


def test_given_back(gpu, clbm_lib):
    out = subprocess.run([sys.executable, "-c", GIVEN_BACK], capture_output=True, text=True, timeout=300,
                         env={**os.environ, "PYTHONPATH": str(PKG)})
    assert out.returncode == 0, out.stderr


def test_threads_with_streams(gpu, clbm_lib):
    W, H, nsnap = 129, 129, 3
    n, g = 9 * W * H, clbm_lib.geom(W, H, 30, 62, 48, 80)
    rng = np.random.default_rng(5)
    f0 = gpu.from_numpy((1 + 0.01 * rng.standard_normal(n)) / 9).cuda()
    snaps = gpu.from_numpy((1 + 0.01 * rng.standard_normal(nsnap * n)) / 9).cuda()
    pre = rng.random(nsnap)
    d = clbm_lib.RunDesc(width=W, height=H, xmin=30, xmax=62, ymin=48, ymax=80, nclones=2, ranks=1, tau=0.56,
                         beta=2e-6, alpha=0.5, force_scale=100.0, dt=0.01)

    def calls(stream, rounds):
        out = []
        for _ in range(rounds):
            with gpu.cuda.stream(stream):
                f = f0.clone()
            clbm_lib.ref_perturbed_state(f.data_ptr(), snaps.data_ptr(), 0.05, nsnap, n, pre, stream.cuda_stream)
            force = clbm_lib.ref_force_on_square(g, f.data_ptr(), 1.7, stream.cuda_stream)
            with clbm_lib.Sampler([d], clbm_lib.FP32, max_steps=2) as s:
                s.init_equilibrium(0, 0.05, 1e-3, 7)
                s.run_interval(2)
                out.append((f.cpu().numpy(), force, s.dump(0, 1)))
            clbm_lib.lib().clbm_destroy(None)
        return out

    gpu.cuda.synchronize()
    want, got = calls(gpu.cuda.Stream(), 1)[0], {}
    streams = [gpu.cuda.Stream() for _ in range(4)]
    threads = [threading.Thread(target=lambda i=i: got.update({i: calls(streams[i], 8)})) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(got) == [0, 1, 2, 3]
    for res in got.values():
        for one in res:
            for a, b in zip(one, want):
                assert np.array_equal(a, b)
