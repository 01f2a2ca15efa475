"""The exact build takes an axis' right node as the left one's neighbour when the
offset in the cell is at least 2^-20 away from 0 and 1 and |x| < 2^10
(pt_axis_exact in csrc/pt_common.cuh).  Here the rule against the reference's
own steps (interpolations.F90:140-149), in IEEE doubles, over grid sizes and
positions that come as close to the rule's edges as they can."""
import numpy as np
import pytest


def _reference(x, d):
    fr = lambda v: v - np.floor(v)
    node = lambda p: np.where((p >= 0) & (p < d), p, 0).astype(np.int64)
    xp = np.float64(d) * fr(x)
    l = np.floor(xp)
    r = node(np.floor(np.float64(d) * fr(x + 1.0 / np.float64(d))))
    return node(l), r, xp - l


@pytest.mark.parametrize("d", [1, 2, 3, 7, 8, 50, 100, 192, 256, 1000, 4097, 65535, 65536, 100003, 262144])
def test_right_node_rule(d):
    rng = np.random.default_rng(d)
    n = 200_000
    cell = rng.integers(0, d, n)
    off = np.concatenate([rng.random(n // 2), 2.0 ** -20 * (1 + rng.random(n // 4) * 4),
                          1 - 2.0 ** -20 * (1 + rng.random(n - n // 2 - n // 4) * 4)])
    x = (cell + off) / d + rng.integers(-1023, 1023, n) * (rng.random(n) < 0.5)
    x = np.concatenate([x, -x, np.nextafter(x, -np.inf), rng.uniform(-1023, 1023, n)])
    l, r, xd = _reference(x, d)
    hi = xd.view(np.int64) >> 32
    rule = (np.abs(x) < 1024) & (hi >= 0x3eb00000) & (hi < 0x3feffffe)
    assert rule.sum() > x.size // 3
    want = np.where(l + 1 == d, 0, l + 1)
    assert np.array_equal(r[rule], want[rule])
