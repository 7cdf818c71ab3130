"""The float64 reciprocal and quotient of the float64 PatchMatch and the per-pixel sweep against exact
rational arithmetic and the division."""
from fractions import Fraction as F

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _device(a, b):
    from py_ortho_b200 import _lib as L
    t = [torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda() for x in (a, b)]
    q, r = torch.empty_like(t[0]), torch.empty_like(t[0])
    L.check(L.load().mvs_debug_quotients(len(a), t[0].data_ptr(), t[1].data_ptr(), q.data_ptr(), r.data_ptr(),
                                         L.stream_handle()))
    return q.cpu().numpy(), r.cpu().numpy()


def _operands(rng, n):
    """Magnitudes that projections meet and far beyond them, both signs, and short mantissas."""
    a = rng.uniform(0.5, 1, n) * 2.0 ** rng.integers(-60, 60, n) * rng.choice([-1, 1], n)
    b = rng.uniform(0.5, 1, n) * 2.0 ** rng.integers(-30, 60, n) * rng.choice([-1, 1], n)
    b[::7] = np.abs(np.round(b[::7], 2)) + 1.0
    a[::5] = np.float32(a[::5])
    b[::11] = 1.0 - 2.0 ** -53 * rng.integers(1, 9, len(b[::11]))     # mantissas near all ones
    b[::13] = 1.0 + 2.0 ** -52 * rng.integers(0, 9, len(b[::13]))     # and near all zeros
    return a, b


def test_reciprocals_are_within_2_to_the_minus_52():
    rng = np.random.default_rng(0)
    a, b = _operands(rng, 20000)
    _, r = _device(a, b)
    assert max(abs(1 - F(x) * F(y)) for x, y in zip(b, r)) <= F(1, 2**52)


def test_quotients_are_the_division_on_random_operands():
    """A random quotient lies within 2^-50 ulp of a midpoint with probability 2^-49."""
    rng = np.random.default_rng(1)
    for _ in range(4):
        a, b = _operands(rng, 4_000_000)
        q, _ = _device(a, b)
        assert np.array_equal(q, a / b)


def test_quotients_near_the_middle_between_two_doubles():
    """a / b = (M + d / B) / 2^54 with odd M: d / (2 B) ulp from the middle between two doubles (B is b's
    mantissa, 2^52 <= B < 2^53). Beyond 2^-50 ulp the result is the division's, within it one of the two."""
    rng = np.random.default_rng(2)
    a, b, d = [], [], []
    while len(a) < 20000:
        B = int(rng.integers(2**51, 2**52)) * 2 + 1
        delta = int(rng.choice([1, 3, 5, 9, 15, 31, 63, 127, 1023])) * (1 if rng.random() < 0.5 else -1)
        M = (-delta * pow(B, -1, 2**54)) % 2**54
        A, rem = divmod(M * B + delta, 2**54)
        assert rem == 0 and M % 2 == 1
        if 2**53 < M and 0 < A < 2**53:
            s = 2.0 ** int(rng.integers(-20, 20))
            a.append(A * s)
            b.append(float(B))
            d.append(abs(delta) / (2 * B))
    a, b, d = np.array(a), np.array(b), np.array(d)
    q, _ = _device(a, b)
    want = a / b
    far = d > 2.0 ** -50
    assert 1000 < far.sum() < len(d) - 1000
    assert np.array_equal(q[far], want[far])
    off = np.abs(q.view(np.int64) - want.view(np.int64))
    assert off.max() <= 1
    print("near ties that round the other way:", int((off > 0).sum()), "of", int((~far).sum()))
