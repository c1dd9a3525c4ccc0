"""Integer model of the fixed-point contraction: the limb cut (rounded, in
range), the 64-bit sums at their largest, and the error against an FP64
multiply-add chain."""
import random
import struct
from fractions import Fraction

import numpy as np
import pytest

CHUNK = 60


def limbs(x, emax):
    """The kernel's steps on 32-bit words: x 2^(56 - e), e = emax - 1022."""
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    bh, bl, m32 = b >> 32, b & 0xFFFFFFFF, 0xFFFFFFFF
    E = (bh >> 20) & 0x7FF
    d = emax - E
    uh, ul = (0x80000000 | (bh << 11) & m32 | (bl >> 21)) & m32, (bl << 11) & m32
    if d >= 32:
        uh, ul = 0, uh
    s = d & 31
    ul, uh = (((uh << 32) | ul) >> s) & m32, uh >> s
    if d >= 64 or E == 0:
        uh = ul = 0
    rl = (ul + 128) & m32
    uh = (uh + (rl < ul)) & m32
    h = ((uh >> 4) + ((uh >> 3) & 1)) & m32
    low = ((((uh << 32) | rl) >> 8) << 4) & m32
    low = (low - (1 << 32) if low >> 31 else low) >> 4
    sg = -1 if bh >> 31 else 0
    return (h ^ sg) - sg, (low ^ sg) - sg


def test_limbs_are_the_rounded_value_and_in_range():
    rng = random.Random(3)
    xs = [rng.choice((-1, 1)) * rng.uniform(0.5, 1) * 2.0 ** rng.randint(-70, 0) for _ in range(20000)]
    xs += [s * (1 - k * 2.0**-53) for s in (-1, 1) for k in (1, 2, 2**23, 2**24, 2**24 + 1, 2**25)]
    xs += [s * (1 - 2.0**-53) for s in (-1, 1)] + [s * 2.0**-k for s in (-1, 1) for k in range(1, 64)] + [0.0, -0.0]
    for x in xs:
        h, low = limbs(x, 1022)  # |x| < 2^0
        assert abs(((h << 28) + low) - Fraction(x) * 2**56) <= Fraction(1, 2)
        assert abs(h) <= 2**28 and abs(low) <= 2**27


def test_sums_fit_64_bits_at_their_largest():
    h, low = limbs(1 - 2.0**-53, 1022)
    assert 2 * CHUNK * max(h, 2**28) ** 2 < 2**63            # re re - im im over a chunk
    assert 4 * CHUNK * max(h, 2**28) * 2**27 < 2**63          # the four cross products
    assert 2 * (CHUNK + 4) * 2**56 >= 2**63                   # and no longer chunk would


@pytest.mark.parametrize("K", [2, 10, 38, 60, 61, 196, 1444])
def test_error_is_no_larger_than_an_fp64_chain(K):
    ld = np.longdouble
    if np.finfo(ld).nmant < 63:
        pytest.skip("no extended precision")
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((24, K)), rng.standard_normal((K, 24))
    ref = A.astype(ld) @ B.astype(ld)
    chain, fx = np.zeros((24, 24)), np.zeros((24, 24))
    for k in range(K):
        chain = (chain.astype(ld) + A[:, k:k + 1].astype(ld) * B[k:k + 1].astype(ld)).astype(float)
    n = -(-K // CHUNK)
    kc = -(-K // n)

    def cut(x, axis):
        e = np.frexp(np.abs(x).max(axis=axis, keepdims=True))[1]
        v = np.rint(np.ldexp(x.astype(ld), 56 - e)).astype(np.int64)
        h = (v + (1 << 27)) >> 28
        return h, v - (h << 28), e

    for k0 in range(0, K, kc):
        (h, low, e), (g, m, f) = cut(A[:, k0:k0 + kc], 1), cut(B[k0:k0 + kc], 0)
        s = (h @ g).astype(ld) * ld(2.0**28) + (h @ m + low @ g).astype(ld)
        fx = fx + np.ldexp(s, e + f - 84).astype(float)
    assert np.linalg.norm((fx - ref).astype(float)) <= np.linalg.norm((chain - ref).astype(float))
