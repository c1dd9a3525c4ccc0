"""Operands of a molecule with spatial symmetry in the FP64 form: elements that the
symmetry forbids are not zero but the noise of earlier roundings, 10^-16 of the others,
and so is every output it forbids.  Three quarters of a tile's outputs then lie below
what exact digits hold and are done by FP64 multiply-adds, a lane a row where many are
marked together, the lanes over k where few are.

The bound of a chain of K multiply-adds is K 2^-53 sum |a||b| for each output; its errors
are about half of 2^-53 sum |a||b| (rms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
U = 2.0**-53


def _check(got, ref, size, K):
    e = (np.abs(got - ref) / (U * size)).astype(float)
    assert e.max() <= K + 4
    assert np.sqrt((e * e).mean()) <= 1.0


def _noisy(x, irreps, noise):
    """x with the elements whose irreps do not multiply to the first one scaled down."""
    g = irreps[0]
    for i in irreps[1:]:
        g = g[..., None] ^ i
    return np.where(g == 0, x, noise * x)


def _t2(rng, io, iv, noise):
    o, v = io.size, iv.size
    t = rng.standard_normal((o, o, v, v)) + 1j * rng.standard_normal((o, o, v, v))
    t = t - t.transpose(1, 0, 2, 3)
    return _noisy(t - t.transpose(0, 1, 3, 2), (io, io, iv, iv), noise)


def _residual(o, v, tei, t):
    from python_code_to_check_c_gb300.engine import CCEngine
    n = o + v
    eng = CCEngine(tei, np.zeros((n, n)), [np.eye(n)], o)
    try:
        got = eng.rhs("CCSD", 1, np.zeros((o, v), complex), t, F=np.zeros((n, n), complex)).cpu().numpy()
        eng.check_errors()
    finally:
        eng.close()
    return got


CASES = pytest.mark.parametrize("o,v,irr,noise", [(7, 31, 4, 1e-16), (7, 31, 2, 1e-12), (10, 38, 8, 1e-16), (6, 33, 4, 1e-7)])


@CASES
def test_ladder(o, v, irr, noise):
    """<ab||ef> t_ijef alone: real by complex."""
    rng = np.random.default_rng(o + v)
    io, iv = rng.integers(0, irr, o), rng.integers(0, irr, v)
    W = rng.standard_normal((v, v, v, v))
    W = W - W.transpose(1, 0, 2, 3)
    W = _noisy(W - W.transpose(0, 1, 3, 2), (iv, iv, iv, iv), noise)
    tei = np.zeros((o + v,) * 4)
    tei[o:, o:, o:, o:] = W
    t = _t2(rng, io, iv, noise)
    got = _residual(o, v, tei, t)
    ab = rng.choice([a * v + b for a in range(v) for b in range(v) if a != b], size=32, replace=False)
    ij = [i * o + j for i in range(o) for j in range(o) if i != j]
    A, B = W.reshape(v * v, v * v)[ab].astype(LD), t.reshape(o * o, v * v)[ij]
    got = got.reshape(o * o, v * v)[np.ix_(ij, ab)]
    for part in (np.real, np.imag):
        b = part(B).astype(LD)
        _check(part(got), 0.5 * (b @ A.T), 0.5 * (np.abs(b) @ np.abs(A).T), v * v)


@CASES
def test_ring(o, v, irr, noise):
    """P(ij) P(ab) t_imae <mb||ej> alone: complex by complex."""
    rng = np.random.default_rng(o * v)
    n = o + v
    io, iv = rng.integers(0, irr, o), rng.integers(0, irr, v)
    W = rng.standard_normal((o, v, v, o))
    W = _noisy(W + W.transpose(3, 2, 1, 0), (io, iv, iv, io), noise)
    tei = np.zeros((n,) * 4)
    tei[:o, o:, o:, :o] = W
    tei[o:, :o, o:, :o] = -W.transpose(1, 0, 2, 3)
    tei[:o, o:, :o, o:] = -W.transpose(0, 1, 3, 2)
    tei[o:, :o, :o, o:] = W.transpose(1, 0, 3, 2)
    t = _t2(rng, io, iv, noise)
    got = _residual(o, v, tei, t)
    w = W.transpose(0, 2, 3, 1).reshape(o * v, o * v)  # (m e), (j b)
    js, bs = rng.choice(o, 3, replace=False), rng.choice(v, 6, replace=False)

    def product(x, y, sign):
        """The four images at j in js, b in bs, all i and a, summed with `sign`."""
        full = (x.transpose(0, 2, 1, 3).reshape(o * v, o * v) @ y).reshape(o, v, o, v)  # i a j b
        full = full.transpose(0, 2, 1, 3)  # i j a b
        r = full + sign * full.transpose(1, 0, 2, 3)
        r = r + sign * r.transpose(0, 1, 3, 2)
        return r[:, js][..., bs]

    live = np.broadcast_to((np.arange(o)[:, None] != js)[:, :, None, None] & (np.arange(v)[:, None] != bs)[None, None],
                           (o, 3, v, 6))
    for part in (np.real, np.imag):
        x, y = part(t).astype(LD), w.astype(LD)
        _check(part(got)[:, js][..., bs][live], product(x, y, -1)[live], product(np.abs(x), np.abs(y), 1)[live], o * v)
