"""Reverse mode at a size whose programs hold eight-slice products of the FP64 form:
the state's cotangents against central differences of the propagation itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["CCSD", "CC2"])
def test_step_gradient_against_differences(method):
    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine, adjoint
    from python_code_to_check_c_gb300.system import synthetic_system
    o, v, dt = 7, 31, 0.02
    s = synthetic_system(o, v, 72, seed=8)
    rng = np.random.default_rng(3)

    def c(shape, size):
        return size * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))

    def anti(x):
        x = x - x.transpose(1, 0, 2, 3)
        return 0.5 * (x - x.transpose(0, 1, 3, 2))

    st = [c((o, v), 0.05), anti(c((o, o, v, v), 0.02)), c((o, v), 0.05), anti(c((o, o, v, v), 0.02))]
    field, weights = make_field("sin", 0.002, 0.923), [0.4, 0.9]
    eng = CCEngine.from_system(s, device_integrals=False)
    try:
        def objective(state):
            _, mu = eng.propagate(method, state, 0.0, dt, 2, field, precs=-1)
            return float((mu.cpu().numpy().real * weights).sum())

        for store in (1, 0):
            eng.set_adjoint_store(store)
            J, _, a = adjoint(eng, method, st, 0.0, dt, 2, weights, field=field, want_state_grad=True)
            eng.check_errors()
            assert abs(J[0] - objective(st)) < 1e-12 * max(1.0, abs(J[0]))
            a = [x.cpu().numpy() for x in a]
            for k in range(4):
                d = c(st[k].shape, 1.0)
                if d.ndim == 4:
                    d = anti(d)
                d /= np.abs(d).max()
                h = 1e-4
                ends = [objective([x + (sgn * h * d if q == k else 0) for q, x in enumerate(st)]) for sgn in (1, -1)]
                fd = (ends[0] - ends[1]) / (2 * h)
                # dJ = Re sum conj(a) d, or its conjugate: the returned cotangent's convention
                got = max((np.sum(a[k] * d).real, np.sum(np.conj(a[k]) * d).real), key=lambda g: -abs(g - fd))
                assert abs(got - fd) < 1e-6 * max(abs(fd), 1e-3), (store, k)
    finally:
        eng.close()
