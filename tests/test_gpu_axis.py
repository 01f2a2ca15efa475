"""The exact build's cell of one axis, pt_axis_exact itself, against the reference's
steps (interpolations.F90:140-149) in IEEE doubles: offsets on both sides of the
rule's edges (2^-20 and 1 - 2^-20 of a cell), positions on both sides of
|x| = 2^10, faces and their neighbours, infinities and NaN."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, d):
    d = np.float64(d)

    def fraction(v):
        return v - np.floor(v)

    def node(p):
        return np.where((p >= 0) & (p < d), p, 0.0).astype(np.int64)    # NaN compares false: 0

    xp = d * fraction(x)
    l = np.floor(xp)
    return node(l), node(np.floor(d * fraction(x + 1.0 / d))), xp - l


def _positions(d):
    rng = np.random.default_rng(d)
    e = 2.0 ** -20
    cells = np.unique(np.concatenate([[0, 1, d // 2, d - 2, d - 1], rng.integers(0, d, 200)]).clip(0, d - 1))
    offs = np.concatenate([[0.0, 2.0 ** -53, e / 2, e, 1.5 * e, 0.25, 0.5, 1 - 1.5 * e, 1 - e, 1 - e / 2, 1 - 2.0 ** -53],
                           rng.random(20), e * (1 + 1e-3 * rng.normal(size=20)), 1 - e * (1 + 1e-3 * rng.normal(size=20))])
    x = ((cells[:, None] + offs[None, :]) / d).ravel()
    shift = np.array([0.0, -1.0, 1.0, 37.0, -512.0, 1022.0, 1023.0, 1024.0, -1023.0, -1024.0, -1025.0, 1e6])
    x = (x[:, None] + shift[None, :]).ravel()
    x = np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf), rng.uniform(-1100, 1100, 20000)])
    special = [0.0, -0.0, 5e-324, -5e-324, -1e-300, 1e-300, -1e-17, 1e300, -1e300, np.inf, -np.inf, np.nan, -np.nan]
    return np.concatenate([x, special])


@pytest.mark.parametrize("d", [1, 2, 3, 8, 50, 100, 256, 1000, 65535, 65536, 100003, 262144])
def test_cell_of_an_axis(cuda, d):
    torch = cuda
    from particles_gb300 import _native as N
    x = _positions(d)
    with np.errstate(invalid="ignore"):
        l, r, xd = _reference(x, d)
    dx = torch.tensor(x, device="cuda")
    gxd = torch.empty(x.size, dtype=torch.float64, device="cuda")
    glr = torch.empty(x.size, 2, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    N.check(N.load().pt_debug_axis(x.size, p(dx), d, p(gxd), p(glr), None), "pt_debug_axis")
    glr, gxd = glr.cpu().numpy(), gxd.cpu().numpy()
    assert np.array_equal(glr[:, 0], l)
    assert np.array_equal(glr[:, 1], r)
    nan = np.isnan(xd)
    assert np.array_equal(np.isnan(gxd), nan)
    assert np.array_equal(gxd[~nan].view(np.int64), xd[~nan].view(np.int64))
