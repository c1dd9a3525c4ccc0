"""The ground-state solver's energies against their formulas, from fewer elements
than the parts of its sums have threads to several passes over them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(2, 3), (3, 9), (7, 13), (9, 23)])
@pytest.mark.parametrize("mode", [0, 1])
def test_energy_of_the_returned_amplitudes(o, v, mode):
    from python_code_to_check_c_gb300.engine import CCEngine
    from python_code_to_check_c_gb300.system import mp2_guess, synthetic_system
    s = synthetic_system(o, v, 3 * (o + v), seed=o * 10 + v)
    tei, f = s.tei(), s.fock
    t2 = mp2_guess(tei, np.linalg.eigh(f)[0], o)
    t1 = 0.01 * np.random.default_rng(o).standard_normal((o, v))
    eng = CCEngine.from_system(s, device_integrals=False)
    try:
        # stops after the first extrapolation, whose energy it returns
        E, it, x1, x2 = eng.ground_state("CCSD", mode, t1, t2, t1, t2, maxsize=3, maxiter=5, E_min=1e300, r_tol=1e-30)
    finally:
        eng.close()
    assert it == 1
    x1, x2 = x1.cpu().numpy(), x2.cpu().numpy()
    g = tei[:o, :o, o:, o:]
    terms = [f[:o, o:] * x1, 0.25 * g * x2]
    if mode == 0:
        terms.append(0.5 * g * x1[:, None, :, None] * x1[None, :, None, :])
    # n terms of either sign, each rounded a few times and added in sums of at most n / 8192 + 45 steps
    tol = sum(np.abs(t).sum() for t in terms) * 2.0**-53 * (4 + o * o * v * v / 8192 + 45)
    assert abs(E - sum(t.sum().real for t in terms)) <= tol
