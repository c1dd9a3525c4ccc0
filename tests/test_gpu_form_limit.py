"""A program of the FP64 form whose packed operands would take more than their limit
keeps the tensor cores for the contractions that gain most, instead of losing them all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_contractions_stay_on_the_tensor_cores():
    import torch

    from oracle.cc_oracle import CCOracle
    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine, profile_step
    from python_code_to_check_c_gb300.system import synthetic_system
    from golden_util import rel_err
    o, v, nb = 10, 38, 240  # L1 would pack 36 GiB
    s = synthetic_system(o, v, 72, seed=6)
    rng = np.random.default_rng(2)

    def c(shape, size):
        return size * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))

    one = [c((o, v), 0.05), c((o, o, v, v), 0.02), c((o, v), 0.05), c((o, o, v, v), 0.02)]
    torch.cuda.empty_cache()
    eng = CCEngine.from_system(s, nb=nb)
    try:
        st = [torch.as_tensor(x, device="cuda").expand((nb,) + x.shape).contiguous() for x in one]
        recs = profile_step(eng, "CCSD", st, 0.0, 0.01, make_field("sin", 0.002, 0.923))
        l1 = [r for r in recs if r["tag"].startswith("ccsd_l1") and r["kind"] == 0]
        deep = [r for r in l1 if r["backend"] == 1]
        assert 0 < len(deep) < len(l1)
        assert sum(r["flops"] for r in deep) > 0.8 * sum(r["flops"] for r in l1)
        got = eng.rhs("CCSD", 2, *st)
        want = CCOracle(s.tei(), o).lam_1eq_rhs(*one, s.fock + 0j)
        for z in (0, nb - 1):
            assert rel_err(got[z].cpu().numpy(), want) < 1e-12
    finally:
        eng.close()
        torch.cuda.empty_cache()
