"""Integer models of what the FP64 form keeps of an operand's small elements: the
fixed-point tiles' limbs and FP32 remainder, the 8-slice products' 8-bit digits."""
import random
import struct
from fractions import Fraction

import numpy as np
import pytest

M32 = 0xFFFFFFFF


def words(x):
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    return b >> 32, b & M32


def f32(bits):
    return float(np.uint32(bits & M32).view(np.float32))


def cut_number(x, emax):
    """The kernel's steps on 32-bit words: limbs h, l, remainder r, x 2^-(emax - 1022)."""
    bh, bl = words(x)
    E = (bh >> 20) & 0x7FF
    d = emax - E
    w = [0, (bl << 11) & M32, (0x80000000 | (bh << 11) | (bl >> 21)) & M32]
    if d >= 32:
        w = [w[1], w[2], 0]
    s = d & 31
    out, ul, uh = (((w[1] << 32) | w[0]) >> s) & M32, (((w[2] << 32) | w[1]) >> s) & M32, w[2] >> s
    rl = (ul + 128) & M32
    uh = (uh + (rl < ul)) & M32
    h = ((uh >> 4) + ((uh >> 3) & 1)) & M32
    low = ((((uh << 32) | rl) >> 8) << 4) & M32
    low = (low - (1 << 32) if low >> 31 else low) >> 4
    t = ((ul << 24) | (out >> 8)) & M32
    r = float(np.float32(t - (1 << 32) if t >> 31 else t)) * 2.0**-32
    f = f32(((126 - d) << 23) | ((bh & 0xFFFFF) << 3) | (bl >> 29)) if 0 <= d <= 125 else 0.0
    if E == 0 or d > 125:
        f = 0.0 if x == 0 else float("nan")
    if E == 0 or d >= 64:
        h = low = 0
        r = f * 2.0**56
    sg = -1 if bh >> 31 else 1
    return sg * h, sg * low, sg * r, sg * f


def test_number_is_its_limbs_and_remainder():
    rng = random.Random(4)
    xs = [rng.choice((-1, 1)) * rng.uniform(0.5, 1) * 2.0**-k for k in range(125) for _ in range(40)]
    xs += [s * (1 - k * 2.0**-53) for s in (-1, 1) for k in (1, 2, 2**23, 2**24 + 1)] + [0.0, -0.0]
    xs += [s * 2.0**-k for s in (-1, 1) for k in range(1, 126)]
    for x in xs:
        h, low, r, f = cut_number(x, 1022)
        assert abs(h) <= 2**28 and -(2**27) <= low <= 2**27 and abs(r) <= 0.5
        v = Fraction(x) * 2**56
        # r is FP32: 2^-24 of itself, and not below 2^-32 where limbs are left
        err = abs(h * 2**28 + low + Fraction(r) - v)
        assert err <= max(abs(Fraction(r)) * Fraction(2) ** -22, Fraction(2) ** -32 if abs(v) >= Fraction(1, 256) else 0)
        assert abs(Fraction(f) - Fraction(x)) <= abs(Fraction(x)) * Fraction(2) ** -23
    assert np.isnan(cut_number(2.0**-130, 1022)[3]) and np.isnan(cut_number(5e-324, 1022)[3])


def digits(x):
    """8 digits of |x| < 1: 7 bits, then 8 bits each, from one biased addition."""
    f = int(abs(Fraction(x)) * 2**63 + Fraction(1, 2)) + 0x0080808080808080
    return [f >> 56] + [((f >> (8 * k)) & 0xFF) - 128 for k in range(6, -1, -1)]


def test_digits_are_the_rounded_value_in_range():
    rng = random.Random(5)
    xs = [rng.uniform(0, 1) * 2.0 ** -rng.randint(0, 70) for _ in range(5000)]
    xs += [1 - 2.0**-53, 0.5, 2.0**-64, 2.0**-65, 0.0, 1 - 2.0**-8, 255 / 256 - 2.0**-53]
    for x in xs:
        d = digits(x)
        assert 0 <= d[0] <= 128 and all(-128 <= q <= 127 for q in d[1:])
        v = sum(Fraction(q, 2 ** (7 + 8 * k)) for k, q in enumerate(d))
        assert abs(v - Fraction(x)) <= Fraction(1, 2**64)


def bf16(bits):
    return f32(bits << 16)


def test_digits_from_bf16_bits():
    """0x4300 + u is the BF16 number 128 + u; the digits' bias is taken from it."""
    for u in range(129):
        assert bf16(0x4300 | u) - 128.0 == u
    for u in range(256):
        assert bf16(0x4300 | (u & 0x7F)) - bf16((u & 0x80) ^ 0x4380) == u - 128


def test_level_sums_are_exact_over_a_chunk():
    """8 slices: the largest sum of a level over a chunk of two K blocks of 64."""
    for level in range(2, 10):
        assert (level - 1) * 128 * 128 * 2 * 64 <= 2**24
    # four levels meet in 64 bits, 4096 K blocks (2048 chunks) of them
    top = sum((p + 1) * 2**21 << (8 * (7 - p)) for p in range(4, 8))
    assert 2048 * top < 2**62


def _rows(kind, K, rng, n=24):
    A, B = rng.standard_normal((n, K)), rng.standard_normal((K, n))
    if kind == "log-normal":
        A, B = A * np.exp(rng.standard_normal((n, K))), B * np.exp(rng.standard_normal((K, n)))
    elif kind == "sparse":
        A, B = A * (rng.random((n, K)) < 0.3), B * (rng.random((K, n)) < 0.3)
    elif kind == "diagonal":
        A = 0.02 * A
        A[:, : min(n, K)] += np.eye(n)[:, : min(n, K)]
    elif kind.startswith("graded"):
        w = float(kind[6:]) ** (-np.arange(K) / (K - 1.0))
        A, B = A * w, B / w[:, None]
    return A, B


@pytest.mark.skipif(np.finfo(np.longdouble).nmant != 63, reason="needs the 64-bit significand (speed)")
@pytest.mark.parametrize("kind", ["normal", "log-normal", "sparse", "diagonal", "graded10", "graded1e2", "graded1e4"])
@pytest.mark.parametrize("K", [38, 200])
def test_eight_slices_leave_less_than_a_multiply_add_chain(kind, K):
    """The outputs that the range guard keeps: rms error against sum |a||b| below 2^-53."""
    rng = np.random.default_rng(len(kind) + K)
    LD = np.longdouble
    A, B = _rows(kind, K, rng)
    ea, eb = np.frexp(np.abs(A).max(1, keepdims=True))[1], np.frexp(np.abs(B).max(0, keepdims=True))[1]

    def cut(x, e):
        v = np.rint(np.ldexp(np.abs(x).astype(LD), 63 - e))
        out = []
        for _ in range(7):
            q = np.floor((v + 128) / 256)
            out.append(np.sign(x) * (v - 256 * q))
            v = q
        return (out + [np.sign(x) * v])[::-1]

    da, db = cut(A, ea), cut(B, eb)
    tot = sum((da[s] @ db[t]) * LD(2) ** (-14 - 8 * (s + t)) for s in range(8) for t in range(8) if s + t <= 7)
    got = np.ldexp(tot, (ea + eb).astype(int)).astype(float)
    S = np.ldexp(np.abs(A), -ea) @ np.ldexp(np.abs(B), -eb)
    keep = S >= 2.0**-10 * np.sqrt(K)
    assert not np.any(got[S == 0])
    size = np.abs(A).astype(LD) @ np.abs(B).astype(LD)
    e = (np.abs(got - A.astype(LD) @ B.astype(LD))[keep] / (size[keep] * 2.0**-53)).astype(float)
    assert kind == "graded1e4" or keep.mean() > 0.9
    if e.size:
        assert np.sqrt((e * e).mean()) < 1.0
