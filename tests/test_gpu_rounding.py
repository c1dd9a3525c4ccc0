"""The update's rounding to decimals, bit for bit numpy's, over the range of
values and decimals: with no integrals, Fock matrix or field a step is the
rounding alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precs", [0, 1, 3, 8, 12, 15, 16, 22])
def test_step_of_nothing_rounds_as_numpy_does(precs):
    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine
    o, v = 6, 40
    n = o + v
    rng = np.random.default_rng(precs)

    def values(shape):
        size = int(np.prod(shape))
        x = rng.standard_normal(size) * 10.0 ** rng.integers(-20, 3, size)
        k = rng.integers(0, 10**6, size) + rng.choice([0.0, 0.5], size)
        x[::3] = (k * 10.0**-precs)[::3]  # multiples and halves of the last decimal
        x[::7] = np.nextafter(x[::7], rng.choice([-np.inf, np.inf], x[::7].shape))
        x[:10] = [0.0, -0.0, 5e-324, -1e-310, 1.0, -1.0, 1e15, 2.0**53, 0.5 * 10.0**-precs, 1.5 * 10.0**-precs]
        return x.reshape(shape)

    st = [values((o, v)) + 1j * values((o, v)), values((o, o, v, v)) + 1j * values((o, o, v, v))] * 2
    eng = CCEngine(np.zeros((n, n, n, n)), np.zeros((n, n)), np.zeros((1, n, n)), o)
    try:
        new, _ = eng.rk4_step("CCSD", st, 0.0, 1e-300, make_field("sin", 0.0, 0.0), precs=precs, with_mu=False)
        for x, y in zip(st, new):
            y = y.cpu().numpy()
            assert np.array_equal(np.around(x.real, precs), y.real) and np.array_equal(np.around(x.imag, precs), y.imag)
    finally:
        eng.close()
