"""Operands whose rows span many powers of two in the FP64 form: every output as
accurate as FP64 multiply-adds leave it, against the sum of its own products'
magnitudes (not against the largest output).

The bound of a chain of K multiply-adds is K 2^-53 sum |a||b|; its errors are about
half of 2^-53 sum |a||b| (rms).  Sums of such contractions add their bounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
U = 2.0**-53


def _check(got, ref, size, K):
    """got: computed; ref, size: exact sums and sums of magnitudes (long double)."""
    live = size > 0
    assert np.array_equal(got[~live], np.zeros_like(got[~live]))
    e = (np.abs(got - ref)[live] / (U * size[live])).astype(float)
    assert e.max() <= K + 4
    assert np.sqrt((e * e).mean()) <= 1.0


# the smaller ones run on the integer pipe, the larger on the tensor cores
@pytest.mark.parametrize("n,nq", [(3, 60), (6, 38), (20, 61), (33, 70), (40, 200)])
@pytest.mark.parametrize("factor", [1e2, 1e4, 1e8, 1e12])
def test_integrals_of_graded_factors(n, nq, factor):
    from python_code_to_check_c_gb300.engine import tei_from_df_device
    rng = np.random.default_rng(n + nq)
    w = factor ** (-np.arange(nq) / (nq - 1.0))
    up = rng.integers(-1, 2, size=(n, n))  # rows that fall, stay and rise along the factors
    B = rng.standard_normal((nq, n, n)) * w[:, None, None] ** up[None]
    got = tei_from_df_device(B).cpu().numpy()

    ps = rng.choice(n, size=3, replace=False)  # these p of <pq||rs>, in extended precision

    def product(x):
        return np.einsum("Qpr,Qqs->pqrs", x[:, ps], x)

    J, S = product(B.astype(LD)), product(np.abs(B).astype(LD))
    off = ~np.eye(n, dtype=bool)
    _check(got[ps][..., off], (J - J.transpose(0, 1, 3, 2))[..., off], (S + S.transpose(0, 1, 3, 2))[..., off], nq)


def _engine(o, v, tei):
    from python_code_to_check_c_gb300.engine import CCEngine
    n = o + v
    return CCEngine(tei, np.zeros((n, n)), [np.eye(n)], o)


def _amplitudes(o, v, w, imag, rng):
    t = rng.standard_normal((o, o, v, v)) + 1j * imag * rng.standard_normal((o, o, v, v))
    t = t - t.transpose(1, 0, 2, 3)
    return (t - t.transpose(0, 1, 3, 2)) / (w[:, None] * w[None, :])


@pytest.mark.parametrize("o,v", [(3, 17), (5, 14), (7, 40)])
@pytest.mark.parametrize("factor,imag", [(1.0, 1e-9), (1e2, 1.0), (1e6, 1.0), (1e6, 1e-9)])
def test_ladder_of_graded_operands(o, v, factor, imag):
    """<ab||ef> t_ijef alone (all other integrals, singles and the Fock matrix are
    zero): real by complex, real and imaginary parts each by itself."""
    rng = np.random.default_rng(o + v)
    n = o + v
    w = factor ** (-np.arange(v) / (v - 1.0))
    W = rng.standard_normal((v, v, v, v))
    W = W - W.transpose(1, 0, 2, 3)
    W = (W - W.transpose(0, 1, 3, 2)) * (w[:, None] * w[None, :])
    tei = np.zeros((n,) * 4)
    tei[o:, o:, o:, o:] = W
    t = _amplitudes(o, v, w, imag, rng)
    eng = _engine(o, v, tei)
    try:
        got = eng.rhs("CCSD", 1, np.zeros((o, v), complex), t, F=np.zeros((n, n), complex)).cpu().numpy()
        eng.check_errors()
    finally:
        eng.close()
    ab = rng.choice([a * v + b for a in range(v) for b in range(v) if a != b], size=24, replace=False)
    ij = [i * o + j for i in range(o) for j in range(o) if i != j]
    A, B = W.reshape(v * v, v * v)[ab].astype(LD), t.reshape(o * o, v * v)[ij]
    got = got.reshape(o * o, v * v)[np.ix_(ij, ab)]
    for part in (np.real, np.imag):
        b = part(B).astype(LD)
        _check(part(got), 0.5 * (b @ A.T), 0.5 * (np.abs(b) @ np.abs(A).T), v * v)


@pytest.mark.parametrize("o,v", [(3, 17), (5, 14), (7, 40)])
@pytest.mark.parametrize("factor,imag", [(1.0, 1e-9), (1e2, 1.0), (1e6, 1.0), (1e6, 1e-9)])
def test_fock_terms_of_graded_operands(o, v, factor, imag):
    """P(ab) F_be t_ijae - P(ij) F_mj t_imab alone: complex by complex."""
    rng = np.random.default_rng(o * v)
    n = o + v
    w = factor ** (-np.arange(v) / (v - 1.0))
    F = np.zeros((n, n), complex)
    F[o:, o:] = (rng.standard_normal((v, v)) + 1j * imag * rng.standard_normal((v, v))) * w[None, :]
    F[:o, :o] = rng.standard_normal((o, o)) + 1j * imag * rng.standard_normal((o, o))
    t = _amplitudes(o, v, w, imag, rng)
    eng = _engine(o, v, np.zeros((n,) * 4))
    try:
        got = eng.rhs("CCSD", 1, np.zeros((o, v), complex), t, F=F).cpu().numpy()
        eng.check_errors()
    finally:
        eng.close()

    def terms(f, x):  # real f, x
        a = np.einsum("ijae,be->ijab", x, f[o:, o:], optimize=False)
        b = np.einsum("imab,mj->ijab", x, f[:o, :o], optimize=False)
        return a, b

    def both(f, x):
        a, b = terms(f, x)
        a = a - a.transpose(0, 1, 3, 2)
        b = b - b.transpose(1, 0, 2, 3)
        return a - b

    def size(f, x):
        a, b = terms(np.abs(f), np.abs(x))
        return a + a.transpose(0, 1, 3, 2) + b + b.transpose(1, 0, 2, 3)

    fr, fi, tr, ti = (x.astype(LD) for x in (F.real, F.imag, t.real, t.imag))
    keep = np.broadcast_to(~np.eye(o, dtype=bool)[:, :, None, None] & ~np.eye(v, dtype=bool)[None, None], t.shape)
    _check(got.real[keep], (both(fr, tr) - both(fi, ti))[keep], (size(fr, tr) + size(fi, ti))[keep], 2 * (o + v))
    _check(got.imag[keep], (both(fr, ti) + both(fi, tr))[keep], (size(fr, ti) + size(fi, tr))[keep], 2 * (o + v))
