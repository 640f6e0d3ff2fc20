"""The branch-free square root of the stage kernels equals the IEEE square root.

Before its last rounding it is off by at most 2^-52 ulp, so it can only round
differently where sqrt(q) lies that close to a midpoint x 2^-53 of two doubles.  With
q 2^106 = Q 2^54 for q in [1, 2) (Q 2^55 in [2, 4)) the distance is
|x^2 - Q 2^54| 2^-107 / m, so the odd x whose squares come within a few units of a
multiple of 2^54 (2^55) are the hardest arguments: they are enumerated here (square
roots modulo a power of two) far beyond that bound, at even exponents of every size,
beside random arguments and the neighbours of exact squares.  Tolerance: none.
"""
import ctypes as C

import numpy as np
import pytest

from boxzyhydro_b200 import _lib


def roots_mod_2k(t, k):
    """The square roots of t (t = 1 mod 8) modulo 2^k."""
    r = 1
    for j in range(3, k):  # r^2 = t mod 2^j  ->  mod 2^(j+1)
        if (r * r - t) >> j & 1:
            r += 1 << (j - 1)
    m = 1 << k
    return sorted({r % m, -r % m, (r + m // 2) % m, (-r + m // 2) % m})


def hard_arguments(reach=4096):
    out = []
    for k, scale in ((54, 1.0), (55, 2.0)):
        for t in range(1 - 8 * (reach // 8), reach, 8):
            for x in roots_mod_2k(t % (1 << k), k):
                for y in (x, x + (1 << k)):
                    if not (1 << 53) <= y < (1 << 54):
                        continue
                    n = y * y - t  # = Q 2^k
                    q = n >> k
                    if n == q << k and (1 << 52) <= q < (1 << 53):
                        out.append(float(q) / 2.0 ** 52 * scale)
    return np.unique(np.array(out))


def test_hard_arguments_are_near_midpoints():
    """The enumeration gives what it says (exact integer arithmetic)."""
    from math import isqrt
    a = hard_arguments(256)
    assert a.size > 60
    for v in a:
        n = int(v * 2.0 ** 52) << 54        # v 2^106
        x = isqrt(n) | 1
        assert min(abs(x * x - n), abs((x - 2) ** 2 - n), abs((x + 2) ** 2 - n)) <= 256


@pytest.mark.gpu
@pytest.mark.parametrize("exp_range,seed", [(2, 1), (120, 2), (900, 3)])
def test_root_is_ieee(exp_range, seed):
    hard = hard_arguments()
    sq = np.random.default_rng(seed).integers(1 << 26, 1 << 27, 4096).astype(float) ** 2
    base = np.concatenate([hard, sq, np.nextafter(sq, np.inf), np.nextafter(sq, 0.0)])
    q = np.concatenate([np.ldexp(base, e) for e in (0, -2, -300, 400)])
    bad, ex = C.c_ulonglong(), C.c_double()
    rc = _lib.lib().bx_check_root(q.ctypes.data_as(C.c_void_p), q.size, 50_000_000, seed,
                                  exp_range, C.byref(bad), C.byref(ex))
    assert rc == 0
    assert bad.value == 0, f"{bad.value} mismatches, e.g. sqrt({ex.value!r})"
