"""The BF16 brick store's records: offset + scale * q with q the value's
(v - offset) / scale in FP64, rounded to FP32 and then to BF16, offset and
scale from the extremes over the records that stencils of the brick reach.

Read back through the force on a fast particle sitting on a node (U = 0, so
f = qom v x B): FP32 evaluation, a few units in the last place; one BF16 step
of q is 2^-9 of the component's half range."""
import numpy as np
import pytest

from test_gpu_bf16 import _accel

pytestmark = pytest.mark.gpu


def _bf16(x):
    b = np.asarray(x, np.float32).view(np.uint32)
    return ((b + 0x7fff + ((b >> 16) & 1)) & 0xffff0000).view(np.float32)


def _stored(a):
    """What the store returns at every node of a (3, d3, d2, d1) field."""
    out = np.empty(a.shape, np.float32)
    _, d3, d2, d1 = a.shape
    reach = lambda b, d: np.arange(b, min(b + 9, d + 1)) % d
    for k in range(0, d3, 8):
        for j in range(0, d2, 8):
            for i in range(0, d1, 8):
                blk = a[:, reach(k, d3)][:, :, reach(j, d2)][:, :, :, reach(i, d1)].reshape(3, -1)
                mn, mx = np.nanmin(blk, 1), np.nanmax(blk, 1)
                off, sc = (0.5 * (mn + mx)).astype(np.float32), (0.5 * (mx - mn)).astype(np.float32)
                sc = np.where(sc > 0, sc, np.float32(1))
                sl = np.s_[:, k:k + 8, j:j + 8, i:i + 8]
                o, s = off[:, None, None, None], sc[:, None, None, None]
                q = ((a[sl] - o.astype(np.float64)) / s.astype(np.float64)).astype(np.float32)
                out[sl] = (s.astype(np.float64) * _bf16(q) + o).astype(np.float32)   # one FMA
    return out


@pytest.mark.parametrize("dm", [(8, 8, 8), (9, 16, 5), (17, 1, 10)])
@pytest.mark.parametrize("kind", ["normal", "mean", "tiny", "huge", "ties", "constant", "nan"])
@pytest.mark.parametrize("with_j", [False, True])
def test_records_at_the_nodes(cuda, dm, kind, with_j):
    torch = cuda
    from particles_gb300 import Fields, params
    d1, d2, d3 = dm
    rng = np.random.default_rng(3)
    b = rng.normal(size=(3, d3, d2, d1))
    if kind == "mean":
        b[0] += 5.0
    elif kind == "tiny":
        b *= 1e-18
    elif kind == "huge":
        b *= 1e18
    elif kind == "ties":                       # offset 0, scale 1, values on BF16 midpoints
        b = rng.integers(-511, 512, b.shape) / 512.0
        b[:, ::4, ::4, ::4] = 1.0
        b[:, 1::4, ::4, ::4] = -1.0
        b[:, -1:, -1:, -1:] = -1.0
    elif kind == "constant":
        b[:] = np.array([0.7, -0.0, 3e-5])[:, None, None, None]
    elif kind == "nan":
        b[1, d3 // 2, 0, d1 // 2] = np.nan
    jj = rng.normal(size=b.shape) if with_j else None
    f = Fields(np.zeros_like(b), b, jj, precision="bf16")
    prm = params.pack_params(qom=1.0, vunit=1.0, tmax=1.0, domain_max=(float(d1), float(d2), float(d3)))
    k, j, i = (a.ravel() for a in np.indices((d3, d2, d1)))
    vec = np.zeros((i.size, 6))
    vec[:, 0], vec[:, 1], vec[:, 2] = i, j, k
    want = _stored(b).reshape(3, -1)
    p = 1000.0
    v = p / np.sqrt(p * p + 1.0)
    near_nan = ~np.isfinite(b)                  # a NaN reaches the stencils next to it
    for ax in (1, 2, 3):
        near_nan |= np.roll(near_nan, -1, ax)
    ok = ~near_nan.any(0).ravel()
    for axis, comp, out, sign in ((0, 1, 5, 1.0), (0, 2, 4, -1.0), (1, 0, 5, -1.0)):
        vec[:, 3:] = 0.0
        vec[:, 3 + axis] = p
        got = _accel(torch, f, prm, vec)[:, out]
        w = sign * v * want[comp].astype(np.float64)
        # v (3 roundings), the store's FMA and the product: 8 units of 2^-24
        assert np.all(np.abs(got - w)[ok] <= 8 * 2.0 ** -24 * np.abs(w)[ok]), (comp, kind)
    f.close()
