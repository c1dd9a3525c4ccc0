"""Which contractions of the FP64 form run on the tensor cores follows from the sizes,
not from the memory that happens to be free when a program is built."""
import numpy as np
import pytest

from golden_util import rel_err

pytestmark = pytest.mark.gpu


def test_form_does_not_depend_on_free_memory():
    import torch

    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine, profile_step
    from python_code_to_check_c_gb300.system import synthetic_system
    o, v = 10, 58
    s = synthetic_system(o, v, 72, seed=6)
    rng = np.random.default_rng(2)

    def c(shape, size):
        return torch.as_tensor(size * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)), device="cuda")

    st = [c((o, v), 0.05), c((o, o, v, v), 0.02), c((o, v), 0.05), c((o, o, v, v), 0.02)]
    tei = torch.as_tensor(s.tei(), device="cuda")

    def run():
        eng = CCEngine(tei, s.fock, s.mu, o)
        try:
            recs = profile_step(eng, "CCSD", st, 0.0, 0.01, make_field("sin", 0.002, 0.923))
            forms = [(r["tag"], r["backend"]) for r in recs]
            return forms, eng.rhs("CCSD", 1, *st).cpu().numpy(), eng.workspace_bytes()
        finally:
            eng.close()

    forms, want, used = run()
    assert any(b == 1 for _, b in forms)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    keep = int(used + 8e8)  # enough for the same system again, not for six of them
    filler = torch.empty(max(free - keep, 0), dtype=torch.uint8, device="cuda")
    try:
        again, got, _ = run()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert again == forms
    assert rel_err(got, want) < 1e-14
