"""Host-buffer runs on the caller's arrays in place (16-byte aligned, pages
shared with the GPU) and through staging (odd alignment; more output rows than a
page holds): the oracle's bits either way, and rows a call does not reach keep
their host values."""
import numpy as np
import pytest

from conftest import small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps", [5, 2100])
@pytest.mark.parametrize("align", ["even", "odd"])
@pytest.mark.parametrize("pinned", [False, True])
def test_host_rows_bitwise(cuda, oracle_lib, nsteps, align, pinned):
    import oracle
    from particles_gb300 import Fields, integrate
    from particles_gb300.integrations import carry_buffer
    npart = 67
    prob = small_problem("rk5", n=10, npart=npart, periods=0.3, seed=91, nsteps=nsteps, tol=1e-7)
    uu, bb = prob["fields"]
    tg = prob["time"]
    so, co, _ = oracle.integrate("rk5", prob["params"], tg, uu, bb, prob["state"].copy())

    def host(a):
        flat = cuda.zeros(a.size + 2, dtype=cuda.float64)
        flat = (flat.pin_memory() if pinned else flat).numpy()
        off = (-(flat.ctypes.data // 8) % 2) + (align == "odd")
        out = flat[off:off + a.size].reshape(a.shape)
        out[:] = a
        assert (out.ctypes.data % 16 == 0) == (align == "even")
        return out

    s = host(prob["state"])
    s[:, 1:] = 7.0                                          # rows not written yet
    f = Fields(host(uu), host(bb))
    cnt, carry = np.zeros((npart, 3), np.int64), carry_buffer(npart)
    half = 0.5 * tg[-1]
    f.integrate("rk5", prob["params"], tg, s, cnt, carry=carry, t_stop=half)
    late = tg > 0.9 * tg[-1]
    assert (s[:, late] == 7.0).all()
    f.integrate("rk5", prob["params"], tg, s, cnt, carry=carry)
    wrote = so[:, :, 6] != 0.0                              # a last row past tmax stays
    assert np.array_equal(cnt, co)
    assert np.array_equal(s[wrote], so[wrote]) and (s[~wrote] == 7.0).all()
    s2 = host(prob["state"])
    _, c2, _ = integrate("rk5", prob["params"], tg, host(uu), host(bb), s2)
    assert np.array_equal(c2, co) and np.array_equal(s2, so)


def test_state_pinned_in_part(cuda, oracle_lib):
    """Only the first pages of the state are registered with the GPU."""
    import mmap
    import oracle
    from particles_gb300 import integrate
    npart = 2 * mmap.PAGESIZE // 64                         # six rows each: twelve pages
    prob = small_problem("rk5", n=10, npart=npart, periods=0.02, seed=92, nsteps=5, tol=1e-6)
    uu, bb = prob["fields"]
    so, co, _ = oracle.integrate("rk5", prob["params"], prob["time"], uu, bb, prob["state"].copy())
    a = prob["state"]
    flat = np.zeros(a.size + mmap.PAGESIZE // 8)
    off = (-flat.ctypes.data % mmap.PAGESIZE) // 8
    s = flat[off:off + a.size].reshape(a.shape)
    s[:] = a
    rt = cuda.cuda.cudart()
    assert int(rt.cudaHostRegister(s.ctypes.data, mmap.PAGESIZE, 0)) == 0
    try:
        _, cnt, _ = integrate("rk5", prob["params"], prob["time"], uu, bb, s)
    finally:
        rt.cudaHostUnregister(s.ctypes.data)
    assert np.array_equal(cnt, co) and np.array_equal(s, so)
