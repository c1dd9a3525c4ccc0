"""Long sums of small elements in the FP64 form: rows whose maximum meets a zero and whose
other elements, 10^-20 of it, meet elements of ordinary size (K = v^2 = 8100).  The
digits under the maximum hold nothing of them, and there are so many that even a floor
under each in what the range guard adds up would have to be far below them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
U = 2.0**-53


def _pairs(x, n):
    """Antisymmetric in its last two indices from its values at e < f."""
    e, f = np.triu_indices(n, 1)
    y = np.zeros(x.shape[:-1] + (n, n), x.dtype)
    y[..., e, f] = x
    y[..., f, e] = -x
    return y


@pytest.mark.parametrize("small", ["integrals", "amplitudes"])
def test_ladder(small):
    from python_code_to_check_c_gb300.engine import CCEngine
    o, v = 3, 90
    n = o + v
    rng = np.random.default_rng(7)
    nab, nij = v * (v - 1) // 2, o * (o - 1) // 2

    def signs(*shape):
        return 1.9 * rng.choice([-1.0, 1.0], size=shape)

    W = _pairs(signs(nab, nab), v)
    t = _pairs(signs(nij, nab) + 1j * signs(nij, nab), v)
    big, zero = (W, t) if small == "integrals" else (t, W)
    big[..., 1:, 1:] *= 1e-20
    zero[..., 0, :] = 0.0
    zero[..., :, 0] = 0.0
    tei = np.zeros((n,) * 4)
    tei[o:, o:, o:, o:] = _pairs(np.moveaxis(W, 0, -1), v).transpose(2, 3, 0, 1)
    t4 = _pairs(np.moveaxis(t, 0, -1), o).transpose(2, 3, 0, 1)
    eng = CCEngine(tei, np.zeros((n, n)), [np.eye(n)], o)
    try:
        got = eng.rhs("CCSD", 1, np.zeros((o, v), complex), t4, F=np.zeros((n, n), complex)).cpu().numpy()
        eng.check_errors()
    finally:
        eng.close()
    a, b = np.triu_indices(v, 1)
    i, j = np.triu_indices(o, 1)
    ab = rng.choice(nab, size=24, replace=False)
    A, B = W[ab].reshape(24, v * v).astype(LD), t.reshape(nij, v * v)
    got = got[i[:, None], j[:, None], a[ab], b[ab]]
    for part in (np.real, np.imag):
        x = part(B).astype(LD)
        size = 0.5 * (np.abs(x) @ np.abs(A).T)
        e = (np.abs(part(got) - 0.5 * (x @ A.T)) / (U * size)).astype(float)
        assert e.max() <= v * v + 4
        assert np.sqrt((e * e).mean()) <= 1.0
