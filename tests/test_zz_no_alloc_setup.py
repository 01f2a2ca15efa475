"""pt_integrate_device_noalloc: a set-up call of one particle on a small grid
readies every later call.  In a process of its own, in which no other call has
loaded a kernel, free device memory stays as that call left it through calls of
either method, small and large."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = r'''
import ctypes as C, sys, time, numpy as np, torch
sys.path.insert(0, "tests")
from conftest import small_problem
from particles_gb300 import _native as N
L = N.load()
few = 80 * torch.cuda.get_device_properties(0).multi_processor_count
p = lambda a: C.c_void_p(a.ctypes.data if isinstance(a, np.ndarray) else a.data_ptr())
calls = []
for method, n, npart in ((1, 4, 1), (1, 8, few + 1), (2, 8, few + 1), (2, 8, 40), (1, 8, 40)):
    pr = small_problem("rk5" if method == 1 else "dop853", n=n, npart=npart, periods=0.01, seed=5, nsteps=2)
    d = [torch.tensor(a, device="cuda") for a in (pr["time"], *pr["fields"], pr["state"])]
    cnt = torch.zeros((npart, 3), dtype=torch.int64, device="cuda")
    calls.append((method, npart, pr, np.array([n] * 3, np.int32), d, cnt))
def call(method, npart, pr, dm, d, cnt):
    t = time.perf_counter()
    N.check(L.pt_integrate_device_noalloc(method, npart, d[0].numel(), p(dm), p(pr["params"]), p(d[0]), p(d[1]),
                                          p(d[2]), p(d[3]), p(cnt), None, None), "noalloc")
    t = time.perf_counter() - t
    assert L.pt_integrate_device_noalloc_check(None) == 0
    return t
torch.cuda.synchronize()
call(*calls[0])
free = torch.cuda.mem_get_info()[0]
times = [call(*c) for c in calls[1:]]
again = [call(*c) for c in calls[1:]]
print("free", free - torch.cuda.mem_get_info()[0], "us", [round(1e6 * t) for t in times], [round(1e6 * t) for t in again])
assert torch.cuda.mem_get_info()[0] == free
for c in calls[1:]:
    assert int(c[5][:, 1].min()) > 0
print("set up once")
'''


def test_a_set_up_call_of_one_particle_readies_later_calls(cuda):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=600)
    print(r.stdout[-2000:])
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "set up once" in r.stdout
