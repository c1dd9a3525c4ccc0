"""The FP64 form's tensor-core contractions (8 slices) where they can go wrong:
ragged tiles and K blocks, every operand type, batches, several K chunks --
against the oracle at the FP64 form's tolerance, with a check that they ran."""
import numpy as np
import pytest

from golden_util import rel_err

pytestmark = pytest.mark.gpu

NAMES = {"CCSD": ("T1eq_rhs", "T2eq_rhs", "lam_1eq_rhs", "lam2eq_rhs"),
         "CC2": ("T1eq_rhs", "T2eq_rhs_CC2", "L1eq_rhs_CC2", "L2eq_rhs_CC2")}


def _case(o, v, nb, scale=1.0):
    from python_code_to_check_c_gb300.system import synthetic_system
    s = synthetic_system(o, v, 72, seed=o * 100 + v)
    rng = np.random.default_rng(o + v + nb)

    def c(shape, size):
        return size * (rng.standard_normal((nb,) + shape) + 1j * rng.standard_normal((nb,) + shape))

    st = [c((o, v), 0.05), c((o, o, v, v), 0.02 * scale), c((o, v), 0.05), c((o, o, v, v), 0.02 * scale)]
    return s, st, s.fock + c((o + v, o + v), 0.01)


def _tensor_core_ops(eng, method, st):
    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import profile_step
    return sum(1 for r in profile_step(eng, method, st, 0.0, 0.01, make_field("sin", 0.002, 0.923)) if r["backend"] == 1)


@pytest.mark.parametrize("o,v,nb", [(7, 31, 1), (5, 45, 1), (9, 33, 3), (12, 26, 2)])
@pytest.mark.parametrize("method", ["CCSD", "CC2"])
def test_residuals_against_the_oracle(o, v, nb, method):
    from oracle.cc_oracle import CCOracle
    from python_code_to_check_c_gb300.engine import CCEngine
    s, st, F = _case(o, v, nb)
    orc = CCOracle(s.tei(), o)
    eng = CCEngine.from_system(s, nb=nb, device_integrals=False)
    try:
        one = [x if nb > 1 else x[0] for x in st]
        assert _tensor_core_ops(eng, method, one) > 0
        for b, name in enumerate(NAMES[method]):
            got = eng.rhs(method, b, *one, F if nb > 1 else F[0]).cpu().numpy().reshape((nb,) + st[b].shape[1:])
            for z in range(nb):
                a = [st[0][z], st[1][z]] + ([st[2][z], st[3][z]] if b > 1 else [])
                assert rel_err(got[z], getattr(orc, name)(*a, F[z])) < 1e-12, (name, z)
        eng.check_errors()
    finally:
        eng.close()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_values_that_digits_cannot_hold(bad):
    """An infinity or a NaN reaches the outputs that the op list takes it to (its
    numpy interpreter gives them) and no others."""
    from oracle.cc_oracle import CCOracle
    from program_emulator import S_F, S_OUT, S_T1, S_T2, S_TEI, Emulator
    from python_code_to_check_c_gb300._lib import program_json
    from python_code_to_check_c_gb300.engine import CCEngine
    o, v = 7, 31
    s, st, F = _case(o, v, 2)
    st[1][1, 0, 1, 2, 3] = bad
    eng = CCEngine.from_system(s, nb=2, device_integrals=False)
    try:
        got = eng.rhs("CCSD", 1, *st, F).cpu().numpy()
    finally:
        eng.close()
    assert rel_err(got[0], CCOracle(s.tei(), o).T2eq_rhs(st[0][0], st[1][0], F[0])) < 1e-12
    e = Emulator(program_json(o, v, "CCSD", 1), o, v)
    nan = st[1][1].copy()
    nan[0, 1, 2, 3] = np.nan  # any product with it is not finite, as with the infinity
    for slot, x in ((S_TEI, s.tei()), (S_T1, st[0][1]), (S_T2, nan), (S_F, F[1]), (S_OUT, np.zeros(nan.shape, complex))):
        e.bind(slot, x)
    e.run()
    want = np.isfinite(e.bufs[S_OUT].reshape(nan.shape))
    assert not want.all() and np.array_equal(np.isfinite(got[1]), want)


@pytest.mark.parametrize("scale", [1e-140, 1e-60, 1e60])
def test_amplitudes_of_unusual_size(scale):
    from oracle.cc_oracle import CCOracle
    from python_code_to_check_c_gb300.engine import CCEngine
    s, st, F = _case(7, 31, 1, scale)
    eng = CCEngine.from_system(s, device_integrals=False)
    try:
        got = eng.rhs("CCSD", 3, *[x[0] for x in st], F[0]).cpu().numpy()
    finally:
        eng.close()
    assert rel_err(got, CCOracle(s.tei(), 7).lam2eq_rhs(*[x[0] for x in st], F[0])) < 1e-12


# the mixed form's bars for 4 and 5 slices; a slice less costs 2^7
@pytest.mark.parametrize("S,tol", [(2, 2**14 * 1e-7), (3, 2**7 * 1e-7), (4, 1e-7), (5, 1e-9)])
@pytest.mark.parametrize("o,v,nb", [(7, 31, 1), (5, 45, 2), (12, 26, 3), (4, 60, 1)])
def test_long_contractions_of_the_mixed_form(o, v, nb, S, tol):
    """K from 3 blocks of 64 (o v) over several exact chunks (v^2), tiles of 96
    and 128 columns with ragged edges, batches, every operand type."""
    from oracle.cc_oracle import CCOracle
    from python_code_to_check_c_gb300.engine import CCEngine
    assert o * v > 128
    s, st, F = _case(o, v, nb)
    orc = CCOracle(s.tei(), o)
    eng = CCEngine.from_system(s, nb=nb, device_integrals=False)
    try:
        eng.set_precision("mixed", S)
        eng.set_tc_policy(0, 1, 1)  # every contraction on the tensor cores
        one = [x if nb > 1 else x[0] for x in st]
        for b, name in enumerate(NAMES["CCSD"]):
            got = eng.rhs("CCSD", b, *one, F if nb > 1 else F[0]).cpu().numpy().reshape((nb,) + st[b].shape[1:])
            for z in range(nb):
                a = [st[0][z], st[1][z]] + ([st[2][z], st[3][z]] if b > 1 else [])
                assert rel_err(got[z], getattr(orc, name)(*a, F[z])) < tol, (name, z)
        eng.check_errors()
    finally:
        eng.close()


def _plain_integrals(B):
    x = np.einsum("Qpr,Qqs->pqrs", B.astype(np.longdouble), B.astype(np.longdouble), optimize=False)
    return x - x.transpose(0, 1, 3, 2)


@pytest.mark.parametrize("n,nq,bad", [(30, 200, None), (33, 100, None), (40, 65, None), (33, 70, np.inf), (32, 130, 5e-324)])
def test_integrals_from_one_packing(n, nq, bad):
    """The symmetric product of the integrals: ragged tiles, the diagonal tiles,
    rows that digits cannot hold; eager and captured (fixed-point tiles) alike."""
    import torch

    from python_code_to_check_c_gb300.engine import tei_from_df_device
    B = np.random.default_rng(n * 1000 + nq).standard_normal((nq, n, n))
    # per product 2^-56 of either maximum for the operands' digits and the levels left out, 2^-53 of the sum
    m = np.abs(B).max()
    tol = 2 * (nq * 3 * 2.0**-56 * m * m + (1 + nq // 60) * 2.0**-53 * nq * m * m)
    if bad is not None:
        B[:, 3, 5] = 0.0
        B[1, 3, 5] = bad
    with np.errstate(all="ignore"):
        ref = _plain_integrals(B)
    ref[..., np.arange(n), np.arange(n)] = 0.0
    Bd = torch.as_tensor(B, device="cuda")
    got = tei_from_df_device(Bd).cpu().numpy()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = tei_from_df_device(Bd)
    g.replay()
    for x in (got, out.cpu().numpy()):
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(x), ok)
        assert np.abs(x[ok] - ref[ok]).max() <= tol
        assert np.array_equal(x[ok], -x.transpose(0, 1, 3, 2)[ok])
