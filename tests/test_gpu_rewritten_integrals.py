"""The FP64 form reads the integrals as they are at each call: a tensor that its
caller writes anew between calls is not answered from operands packed before."""
import numpy as np
import pytest

from golden_util import rel_err

pytestmark = pytest.mark.gpu


def _system(seed):
    from python_code_to_check_c_gb300.system import synthetic_system
    return synthetic_system(7, 31, 72, seed=seed)


def _state(o, v):
    rng = np.random.default_rng(9)

    def c(shape, size):
        return size * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))

    return [c((o, v), 0.05), c((o, o, v, v), 0.02), c((o, v), 0.05), c((o, o, v, v), 0.02)]


def _calls(eng, st, F):
    """Every kind of call that reads the integrals, results as host arrays."""
    import torch

    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import adjoint
    field = make_field("sin", 0.002, 0.923)
    out = [eng.rhs(m, b, *st, F=F) for m in ("CCSD", "CC2") for b in range(4)]
    new, mu = eng.rk4_step("CCSD", st, 0.0, 0.01, field)
    out += list(new) + [mu]
    new, mu = eng.propagate("CCSD", st, 0.0, 0.01, 3, field)
    out += list(new) + [mu]
    E, _, x1, x2 = eng.ground_state("CCSD", 0, 0 * st[0], 0 * st[1], maxsize=3, maxiter=2, E_min=0.0)
    out += [torch.tensor([E]), x1, x2]
    J, gE, a = adjoint(eng, "CCSD", st, 0.0, 0.01, 2, [0.3, 0.7], field=field, want_state_grad=True)
    out += [torch.as_tensor(J), torch.as_tensor(gE)] + list(a)
    return [x.cpu().numpy() for x in out]


def test_integrals_written_anew_between_calls():
    import torch

    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine, profile_step
    a, b = _system(1), _system(2)
    st = _state(7, 31)
    ea, eb = (CCEngine(s.tei(), a.fock, a.mu, a.o) for s in (a, b))
    try:
        recs = profile_step(ea, "CCSD", st, 0.0, 0.01, make_field("sin", 0.002, 0.923))
        assert any(r["backend"] == 1 for r in recs)  # some contractions run on packed operands
        want = _calls(eb, st, a.fock + 0j)
        first = _calls(ea, st, a.fock + 0j)
        ea.tei.copy_(torch.as_tensor(b.tei(), device="cuda"))
        for x, y, z in zip(_calls(ea, st, a.fock + 0j), want, first):
            assert rel_err(x, y) < 1e-12
            assert np.array_equal(z, y) or rel_err(z, y) > 1e-6  # (the first integrals gave something else)
    finally:
        ea.close()
        eb.close()


def test_captured_residual_reads_the_integrals_at_replay():
    import torch

    from python_code_to_check_c_gb300.engine import CCEngine
    a, b = _system(3), _system(4)
    st = [torch.as_tensor(x, device="cuda") for x in _state(7, 31)]
    F = torch.as_tensor(a.fock + 0j, device="cuda")
    ea, eb = (CCEngine(s.tei(), a.fock, a.mu, a.o) for s in (a, b))
    try:
        ea.rhs("CCSD", 1, *st, F=F)  # builds the program
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = ea.rhs("CCSD", 1, *st, F=F)
        ea.tei.copy_(torch.as_tensor(b.tei(), device="cuda"))
        g.replay()
        assert rel_err(out.cpu().numpy(), eb.rhs("CCSD", 1, *st, F=F).cpu().numpy()) < 1e-12
    finally:
        ea.close()
        eb.close()
