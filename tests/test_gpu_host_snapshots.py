"""A snapshot in host arrays -- packed in place (16-byte aligned; BF16 up to 64^3
nodes) or from a staged copy, pinned or not -- gives the store that the same
snapshot in device arrays gives: forces at random points, bit for bit."""
import numpy as np
import pytest

from test_gpu_mixed import _accel_on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dm", [(1, 1, 1), (9, 16, 7), (64, 64, 64), (64, 64, 65)])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("with_j", [False, True])
def test_host_snapshot_gives_the_device_store(cuda, dm, precision, with_j):
    torch = cuda
    from particles_gb300 import Fields, params
    rng = np.random.default_rng(sum(dm))
    arrays = [rng.normal(size=(3, dm[2], dm[1], dm[0])) for _ in range(3 if with_j else 2)]
    prm = params.pack_params(qom=200.0, vunit=0.05, tmax=1.0, dtmax=1.0, atol=1e-8, rtol=1e-8)
    vec = np.concatenate([rng.random((5000, 3)), rng.normal(size=(5000, 3))], axis=1)

    def force(make):
        f = Fields(*[make(a) for a in arrays], precision=precision)
        out = _accel_on_device(torch, f, prm, vec)
        f.close()
        return out.view(np.int64)

    def host(off, pinned):
        def make(a):
            flat = torch.zeros(a.size + 2, dtype=torch.float64, pin_memory=pinned).numpy()
            off_ = (-(flat.ctypes.data // 8) % 2) + off
            v = flat[off_:off_ + a.size].reshape(a.shape)
            v[:] = a
            return v
        return make

    want = force(lambda a: torch.tensor(a, device="cuda"))
    for off in (0, 1):
        for pinned in (False, True):
            assert np.array_equal(force(host(off, pinned)), want), (off, pinned)
