"""The two rules by which the face geometry of EPA leaves FP64 operations out, against the full
arithmetic in NumPy doubles (the device evaluates the same operations unfused): the signs of a
face's barycentric weights from their numerators, and the reliability test of a face normal from
the larger product instead of the error sum.  A rule may ask for the full arithmetic; where
it does not, the answers must agree exactly."""
import numpy as np
import pytest


def exponent(x):
    return ((x.view(np.int64) >> 52) & 0x7FF).astype(np.int64)


def faces(scale, flat, seed, n=200_000):
    rng = np.random.default_rng(seed)
    p = rng.normal(0, 1, (3, n, 3))
    p[:, :, 1] *= flat  # nearly in one plane with the origin
    p[:, : n // 8] = np.round(p[:, : n // 8] * 2) / 2  # exact zeros and ties
    p[2, n // 8: n // 4] = p[0, n // 8: n // 4] * rng.uniform(0, 1, (n // 8, 1)) + 1e-7 * p[1, n // 8: n // 4]
    s = (p * scale).astype(np.float32)
    s[np.abs(s) < 1e-30] = 0  # the coordinates the solver accepts are zero or within 1e-30 .. 1e30
    return s.astype(np.float64)


@pytest.mark.parametrize("scale", [1e-20, 1e-3, 1.0, 1e3, 1e20])
@pytest.mark.parametrize("flat", [0.0, 1e-6, 1.0])
def test_rules_agree_with_the_full_arithmetic(scale, flat):
    a, b, c = faces(scale, flat, seed=int(np.log10(scale)) + 40)
    u, v = a - b, a - c
    with np.errstate(all="ignore"):
        s = u[:, [1, 2, 0]] * v[:, [2, 0, 1]]
        t = u[:, [2, 0, 1]] * v[:, [1, 2, 0]]
        raw = s - t
        ns = np.abs(raw).max(1)
        bound = 2.0**-49 * (np.abs(s) + np.abs(t)).max(1)
        big = np.maximum(np.abs(s), np.abs(t)).max(1)
        surely = ns > np.maximum(big * 2.0**-28, 0)
        assert not (surely & ~(ns > 2.0**20 * bound)).any()

        ok = (ns > 0) & np.isfinite(ns)
        sn = raw / ns[:, None]
        dot = lambda x, y: (x[:, 0] * y[:, 0] + x[:, 1] * y[:, 1]) + x[:, 2] * y[:, 2]
        cross = lambda x, y: x[:, [1, 2, 0]] * y[:, [2, 0, 1]] - x[:, [2, 0, 1]] * y[:, [1, 2, 0]]
        nsq = dot(sn, sn)
        n0, n1 = dot(cross(u, a), sn), dot(cross(a, v), sn)
        gamma, beta = n0 / nsq / ns, n1 / nsq / ns
        alpha = 1.0 - gamma - beta
        den = ns * nsq
        rest = den - (n0 + n1)
        e = exponent(ns)
        terms = np.maximum(exponent(den), np.maximum(exponent(n0), exponent(n1)))
        sure = ok & (e > 823) & (e < 1223) & (exponent(rest) + 40 > terms)
    assert sure.any() or flat == 0.0
    for full, short in ((gamma, n0), (beta, n1), (alpha, rest)):
        assert np.isfinite(full[sure]).all()
        assert np.array_equal(full[sure] < 0, short[sure] < 0)
