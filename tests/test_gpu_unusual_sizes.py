"""Amplitudes far from one in the FP64 form, in a residual that consists of them alone:
what a contraction makes of them sets the size of the result, so that a product dropped,
flushed or scaled wrongly shows.

<ab||ef> t_ijef with all other integrals, the singles and the Fock matrix zero; the bound
is that of K FP64 multiply-adds for each output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
U = 2.0**-53


# the smaller one runs on the integer pipe, the larger on the tensor cores
@pytest.mark.parametrize("o,v", [(3, 17), (7, 40)])
@pytest.mark.parametrize("k", [-960, -800, -465, -200, 200, 900])
def test_ladder_of_scaled_amplitudes(o, v, k):
    from python_code_to_check_c_gb300.engine import CCEngine
    rng = np.random.default_rng(o + v)
    n = o + v
    W = rng.standard_normal((v, v, v, v))
    W = W - W.transpose(1, 0, 2, 3)
    W = W - W.transpose(0, 1, 3, 2)
    tei = np.zeros((n,) * 4)
    tei[o:, o:, o:, o:] = W
    t = rng.standard_normal((o, o, v, v)) + 1j * rng.standard_normal((o, o, v, v))
    t = t - t.transpose(1, 0, 2, 3)
    t = t - t.transpose(0, 1, 3, 2)
    eng = CCEngine(tei, np.zeros((n, n)), [np.eye(n)], o)
    try:
        got = eng.rhs("CCSD", 1, np.zeros((o, v), complex), t * 2.0**k, F=np.zeros((n, n), complex)).cpu().numpy()
        eng.check_errors()
    finally:
        eng.close()
    ab = rng.choice([a * v + b for a in range(v) for b in range(v) if a != b], size=24, replace=False)
    ij = [i * o + j for i in range(o) for j in range(o) if i != j]
    A, B = W.reshape(v * v, v * v)[ab].astype(LD), t.reshape(o * o, v * v)[ij]
    got = got.reshape(o * o, v * v)[np.ix_(ij, ab)]
    for part in (np.real, np.imag):
        b = part(B).astype(LD)
        size = 0.5 * (np.abs(b) @ np.abs(A).T)
        e = (np.abs(np.ldexp(part(got), -k) - 0.5 * (b @ A.T)) / (U * size)).astype(float)
        assert e.max() <= v * v + 4
        assert np.sqrt((e * e).mean()) <= 1.0
