"""The fixed-point contraction kernel where it can go wrong: edges of tiles and
K chunks, operands at the ends of the exponent range, infinities and NaNs."""
import numpy as np
import pytest

from golden_util import rel_err

pytestmark = pytest.mark.gpu


def _tei(B):
    from python_code_to_check_c_gb300.engine import tei_from_df_device
    return tei_from_df_device(B).cpu().numpy()


def _plain(B):
    x = np.einsum("Qpr,Qqs->pqrs", B.astype(np.longdouble), B.astype(np.longdouble))
    return x - x.transpose(0, 1, 3, 2)


@pytest.mark.parametrize("n,nq", [(1, 1), (2, 59), (3, 60), (4, 61), (5, 7), (8, 121), (9, 180), (13, 33)])
def test_real_contraction_edges(n, nq):
    B = np.random.default_rng(n * 1000 + nq).standard_normal((nq, n, n))
    # a product is off by at most 2^-56 of either maximum and 2^-58 of both, a chunk's sum by 2^-53 of itself
    m = np.abs(B).max()
    tol = 2 * (nq * 3 * 2.0**-56 * m * m + (1 + nq // 60) * 2.0**-53 * nq * m * m)
    assert np.abs(_tei(B) - _plain(B)).max() <= tol


@pytest.mark.parametrize("scale", [1e-150, 1e-145, 1e145, 1e152])
def test_scales_at_the_ends_of_the_range(scale):
    B = np.random.default_rng(5).standard_normal((70, 4, 4)) * scale
    ref = _plain(B)
    assert rel_err(_tei(B) / scale**2, (ref / np.longdouble(scale) ** 2).astype(float)) < 1e-14


def test_values_just_below_a_power_of_two():
    rng = np.random.default_rng(8)
    k = rng.choice([1, 2, 2**23, 2**24, 2**24 + 1, 2**25], size=(64, 4, 4))
    B = rng.choice([-1.0, 1.0], size=(64, 4, 4)) * (1 - k * 2.0**-53)
    assert np.abs(_tei(B) - _plain(B)).max() <= 2 * 64 * (3 * 2.0**-56 + 2.0**-53)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e300, 5e-324])
def test_unusual_values_do_what_fp64_does(bad):
    B = np.random.default_rng(6).standard_normal((64, 5, 5))
    B[7, 1, 2] = bad
    B[40, 3, 3] = 0.0
    with np.errstate(all="ignore"):
        x = np.einsum("Qpr,Qqs->pqrs", B, B)
        ref = x - x.transpose(0, 1, 3, 2)
    ref[..., np.arange(5), np.arange(5)] = 0.0  # the diagonal r = s is written as zero
    got = _tei(B)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref)) and np.array_equal(np.isnan(got), np.isnan(ref))
    ok = np.isfinite(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-13 * max(1.0, np.abs(ref[ok]).max())


@pytest.mark.parametrize("o,v,nb", [(1, 1, 1), (1, 17, 2), (2, 16, 1), (3, 33, 1), (5, 15, 3)])
@pytest.mark.parametrize("method", ["CCSD", "CC2"])
def test_residuals_at_ragged_sizes(o, v, nb, method):
    from oracle.cc_oracle import CCOracle
    from python_code_to_check_c_gb300.engine import CCEngine
    from python_code_to_check_c_gb300.system import synthetic_system
    s = synthetic_system(o, v, 3 * (o + v), seed=77 + o)
    rng = np.random.default_rng(o + v)

    def c(shape, size):
        return size * (rng.standard_normal((nb,) + shape) + 1j * rng.standard_normal((nb,) + shape))

    st = [c((o, v), 0.1), c((o, o, v, v), 0.05), c((o, v), 0.1), c((o, o, v, v), 0.05)]
    F = s.fock + c((o + v, o + v), 0.01)
    orc = CCOracle(s.tei(), o)
    names = {"CCSD": ("T1eq_rhs", "T2eq_rhs", "lam_1eq_rhs", "lam2eq_rhs"),
             "CC2": ("T1eq_rhs", "T2eq_rhs_CC2", "L1eq_rhs_CC2", "L2eq_rhs_CC2")}[method]
    eng = CCEngine.from_system(s, nb=nb, device_integrals=False)
    try:
        for b, name in enumerate(names):
            args = [x if nb > 1 else x[0] for x in st] + [F if nb > 1 else F[0]]
            got = eng.rhs(method, b, *args).cpu().numpy().reshape((nb,) + st[b].shape[1:])
            for z in range(nb):
                a = [st[0][z], st[1][z]] + ([st[2][z], st[3][z]] if b > 1 else [])
                assert rel_err(got[z], getattr(orc, name)(*a, F[z])) < 1e-12, (name, z)
    finally:
        eng.close()


def test_small_systems_on_several_threads_and_streams():
    """The one-launch phases of several engines at a time: each has its own barrier and temporaries."""
    import threading

    import torch

    from python_code_to_check_c_gb300._lib import make_field
    from python_code_to_check_c_gb300.engine import CCEngine
    from python_code_to_check_c_gb300.system import mp2_guess, synthetic_system
    sizes = [(3, 5), (4, 8), (2, 7), (4, 6)]
    field, jobs, got, errors = make_field("sin", 0.002, 0.923), [], {}, []

    def work(k):
        eng, st, stream = jobs[k]
        with torch.cuda.stream(stream):
            fin, mu = eng.propagate("CCSD", st, 0.0, 0.01, 40, field)
            res = [mu] + list(fin) + [eng.rhs("CCSD", b, *st) for b in range(4)]
            eng.check_errors()
            return [x.cpu().numpy() for x in res]

    def thread(k):
        try:
            got[k] = [work(k) for _ in range(5)]
        except Exception as ex:  # noqa: BLE001 - reported by the main thread
            errors.append(ex)

    for k, (o, v) in enumerate(sizes):
        s = synthetic_system(o, v, 40, seed=9 + k)
        t1, t2 = np.full((o, v), 0.01 + 0.002j), mp2_guess(s.tei(), s.eps(), o) + 0j
        jobs.append((CCEngine.from_system(s, device_integrals=False), (t1, t2, t1, t2), torch.cuda.Stream()))
    want = [work(k) for k in range(len(sizes))]  # builds the programs and captures the steps
    ts = [threading.Thread(target=thread, args=(k,)) for k in range(len(sizes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for k in range(len(sizes)):
        for run in got[k]:
            for a, b in zip(want[k], run):
                assert rel_err(b, a) < 1e-12
        jobs[k][0].close()
