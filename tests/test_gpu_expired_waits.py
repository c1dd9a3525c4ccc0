"""A bounded wait that runs out leaves NaN and a recorded error, never numbers of an
earlier call: the grid barrier of the one-launch phases, the tensor-core kernel's
barriers (every wait given up at once, so nothing is left in flight)."""
import numpy as np
import pytest

from golden_util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v,block", [(3, 5, 0), (4, 8, 1), (4, 8, 3), (7, 31, 1), (7, 31, 3)])
def test_expired_wait_leaves_nan(o, v, block):
    from python_code_to_check_c_gb300 import _lib
    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine
    from python_code_to_check_c_gb300.system import synthetic_system
    s = synthetic_system(o, v, 72, seed=5)
    rng = np.random.default_rng(1)

    def c(shape, size):
        return size * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))

    st = [c((o, v), 0.05), c((o, o, v, v), 0.02), c((o, v), 0.05), c((o, o, v, v), 0.02)]
    F = s.fock + c((o + v, o + v), 0.01)
    field = make_field("sin", 0.002, 0.923)
    eng = CCEngine.from_system(s, device_integrals=False)
    try:
        want = eng.rhs("CCSD", block, *st, F=F).cpu().numpy()
        eng.check_errors()
        assert eng.lib.tdcc_set_wait_limit(eng.handle, -1) == 0
        got = eng.rhs("CCSD", block, *st, F=F).cpu().numpy()
        assert np.isnan(got).all()
        with pytest.raises(_lib.TdccError, match="gave up"):
            eng.check_errors()
        with pytest.raises(_lib.TdccError):  # the dipole is not finite
            eng.propagate("CCSD", st, 0.0, 0.01, 2, field)
        assert eng.lib.tdcc_set_wait_limit(eng.handle, 0) == 0
        for _ in range(20):  # clears the flags, a program at a time
            try:
                eng.check_errors()
                break
            except _lib.TdccError:
                pass
        again = eng.rhs("CCSD", block, *st, F=F).cpu().numpy()
        assert rel_err(again, want) < 1e-14
        eng.check_errors()
        state, mu = eng.propagate("CCSD", st, 0.0, 0.01, 2, field)
        assert np.isfinite(mu.cpu().numpy()).all()
        eng.check_errors()
    finally:
        eng.close()
