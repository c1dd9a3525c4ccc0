"""What a user of the engine has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (``CCEngine``, ``adjoint``,
``spectrum``, ``tei_from_df_device``).  ``exact`` restates the equations in plain torch,
complex128, one trajectory at a time.  Sizes are those of the repository's workloads and
tests (o = 3..18 occupied, v = 5..82 virtual spin orbitals) and ragged ones between them."""
import math
import random

import numpy as np
import torch

from python_code_to_check_c_gb300._lib import make_field
from python_code_to_check_c_gb300.engine import CCEngine, adjoint, tei_from_df_device
from python_code_to_check_c_gb300.spectrum import spectrum
from python_code_to_check_c_gb300.system import synthetic_system

A0, W0 = 0.002, 0.923  # the field E(t) = A sin(w0 t) of the repository's runs
BLOCKS = ("T1", "T2", "L1", "L2")


def listed():
    def rhs(name, method, block, o, v, nq, slices=0, nb=1):
        return dict(name=name, kind="rhs", method=method, block=block, o=o, v=v, nq=nq, slices=slices, nb=nb)

    return [
        # the smallest call: one residual of a system of a few orbitals (host and launch latency)
        rhs("t1_rhs_o3_v5_fp64", "CCSD", "T1", 3, 5, 24),
        # one step of the loop body on a small system, step by step as a caller with its own loop does
        dict(name="step_cc2_o4_v8_fp64", kind="step", method="CC2", o=4, v=8, nq=40, slices=0, nb=1),
        # minimal-basis water: the device-resident loop in the default precision
        dict(name="propagate_o10_v14_fp64", kind="propagate", method="CCSD", o=10, v=14, nq=72, slices=0, nb=1, steps=8),
        # double-zeta water, default precision: the largest T residual of a step
        rhs("t2_rhs_o10_v38_fp64", "CCSD", "T2", 10, 38, 144),
        # a ragged size, the approximate method's Lambda residual
        rhs("l1_rhs_cc2_o9_v31_fp64", "CC2", "L1", 9, 31, 144),
        # batched trajectories in the mixed form: the largest Lambda residual of their step
        rhs("l2_rhs_o10_v38_mixed4_x24", "CCSD", "L2", 10, 38, 144, slices=4, nb=24),
        # the production run: 24 trajectories of double-zeta water, mixed form
        dict(name="propagate_o10_v38_mixed4_x24", kind="propagate", method="CCSD", o=10, v=38, nq=144, slices=4, nb=24,
             steps=2),
        # the largest system of the uneven batch, with the slices that strong integrals need
        rhs("t2_rhs_o18_v82_mixed5", "CCSD", "T2", 18, 82, 144, slices=5),
        # backward: a pulse gradient through the propagation
        dict(name="gradient_o6_v12_fp64", kind="gradient", method="CCSD", o=6, v=12, nq=72, slices=0, nb=1, steps=8),
        # ground state by DIIS before a propagation
        dict(name="ground_o10_v14_fp64", kind="ground", method="CCSD", o=10, v=14, nq=72, iters=12),
        # post-processing: the dipole spectrum of a 2000-step run
        dict(name="spectrum_2000", kind="spectrum", steps=2000),
        # preparation of a system: the integrals from the density-fitting factors
        dict(name="integrals_n48_q144", kind="integrals", o=10, v=38, nq=144),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    top = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(("rhs", "rhs", "rhs", "rhs", "step", "propagate", "propagate", "gradient", "ground", "spectrum",
                           "integrals"))
        if kind == "spectrum":
            return dict(kind=kind, steps=_log(rng, 200, 20000))
        c = dict(kind=kind, method=rng.choice(("CCSD", "CCSD", "CC2")))
        if kind in ("rhs", "propagate", "step"):
            c["slices"] = rng.choice((0, 0, 4, 5))
            c["o"] = _log(rng, 6, 18) if c["slices"] else _log(rng, 2, 14)
            c["v"] = _log(rng, max(c["o"], 12), 82) if c["slices"] else _log(rng, max(c["o"], 4), 58)
            c["nb"] = rng.choice((1, 1, 3, 8, 24))
            c["nq"] = 3 * (c["o"] + c["v"])
            if kind == "rhs":
                c["block"] = rng.choice(BLOCKS)
            elif kind == "propagate":
                c["steps"] = rng.randint(2, 8)
            # the plain-torch restatement of a case stays within seconds, its workspace on the card
            if (c["nb"] > 1 and c["o"] * c["v"] > 400) or (kind != "rhs" and c["nb"] * c.get("steps", 1) * c["o"] * c["v"] > 20000):
                continue
        elif kind == "integrals":
            c = dict(kind=kind, o=_log(rng, 4, 18), v=_log(rng, 18, 82), nq=_log(rng, 40, 200))
        elif kind == "gradient":
            c.update(o=_log(rng, 3, 8), v=_log(rng, 8, 20), slices=0, nb=1, steps=rng.randint(4, 10))
            c["nq"] = 3 * (c["o"] + c["v"])
        else:  # ground: a system small enough for DIIS to converge on the seeded integrals
            c.update(o=_log(rng, 3, 10), v=_log(rng, 8, 16), nq=72, iters=rng.randint(9, 13))
        if c.get("nq", 0) > 240 or work(c)["flops"] > top:
            continue
        return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _tei(B):
    """<pq||rs> = (pr|qs) - (ps|qr), (pr|qs) = sum_Q B_Qpr B_Qqs, in plain torch."""
    nq, n, _ = B.shape
    Bm = B.reshape(nq, n * n)
    J = (Bm.T @ Bm).reshape(n, n, n, n).permute(0, 2, 1, 3)
    return (J - J.transpose(2, 3)).contiguous()


def _mp2(tei, fock, o):
    e = torch.diagonal(fock)
    d = (e[:o, None, None, None] + e[None, :o, None, None] - e[None, None, o:, None] - e[None, None, None, o:])
    return tei[:o, :o, o:, o:] / d


def _inputs(case, seed):
    """Integrals, Fock matrix, dipoles and amplitudes near a ground state, on the GPU."""
    o, v, nb = case["o"], case["v"], case.get("nb", 1)
    s = synthetic_system(o, v, case["nq"], seed=1000 * seed + 7 * o + v, all_dipoles=True)
    dev = torch.device("cuda")
    # at twice the minimal-basis size and beyond, the factors are scaled so that the correlation stays
    # as strong as at that size
    scale = min(1.0, math.sqrt(24.0 / (o + v)))
    B = torch.as_tensor(s.B, device=dev) * scale
    tei = _tei(B)
    fock = torch.as_tensor(s.fock, device=dev)
    mu = [torch.as_tensor(m, device=dev) for m in s.mu]
    g = torch.Generator(device=dev).manual_seed(1234567 + seed)
    t2 = _mp2(tei, fock, o)

    def noise(shape, size):
        x = torch.randn((nb,) + shape + (2,), dtype=torch.float64, device=dev, generator=g) * size
        return torch.view_as_complex(x)

    def anti(x):
        x = x - x.transpose(-1, -2)
        return 0.5 * (x - x.transpose(-3, -4))

    amp = float(t2.abs().mean()) + 1e-12
    st = []
    for _ in range(2):
        st.append(noise((o, v), 0.01))
        st.append(t2.to(torch.complex128) + anti(noise((o, o, v, v), 0.1 * amp)))
    return dict(B=B, tei=tei, fock=fock, mu=mu, state=[x[0].contiguous() if nb == 1 else x.contiguous() for x in st])


def _fields(case):
    """(polarisation, A, w0) of every trajectory of a batched run."""
    amps, ws = (0.001, 0.002, 0.005, 0.01), (0.5, 0.923)
    return [(k % 3, amps[(k // 3) % 4], ws[(k // 12) % 2]) for k in range(case["nb"])]


def _dressed(case, d):
    """The dressed Fock matrices a residual call of each trajectory sees."""
    E = [0.7 * A for _, A, _ in _fields(case)] if case["nb"] > 1 else [0.7 * A0]
    F = torch.stack([d["fock"] - e * d["mu"][2] for e in E]).to(torch.complex128)
    return F[0].contiguous() if case["nb"] == 1 else F


def prepare(case, seed):
    kind = case["kind"]
    if kind == "spectrum":
        dev, n = torch.device("cuda"), case["steps"]
        r = np.random.default_rng(seed)
        t = torch.arange(n, dtype=torch.float64, device=dev) * 0.005
        mu = torch.zeros(n, dtype=torch.complex128, device=dev)
        for w, a in zip(r.uniform(0.2, 3.0, 6), r.uniform(1e-4, 1e-2, 6)):  # the induced dipole's lines
            mu += torch.complex(a * torch.sin(w * t), 1e-4 * a * torch.cos(w * t))
        return dict(case=case, mu=mu + r.uniform(0.01, 0.1))
    d = _inputs(case, seed)
    if kind == "integrals":
        return dict(case=case, B=d["B"])
    # the engine as a running program has it: programs built, workspaces laid out
    eng = CCEngine(d["tei"], d["fock"], d["mu"], case["o"], nb=case.get("nb", 1))
    if case.get("slices"):
        eng.set_precision("mixed", case["slices"])
    s = dict(case=case, eng=eng, state=d["state"])
    if kind == "rhs":
        s["F"] = _dressed(case, d)
    elif kind in ("step", "propagate"):
        s["field"] = make_field("sin", A0, W0)
        if case["nb"] > 1:
            f = _fields(case)
            eng.set_fields([make_field("sin", A, w) for _, A, w in f], [p for p, _, _ in f])
            s["field"] = None
    elif kind == "gradient":
        s["field"] = make_field("sin", A0, W0)
        s["weights"] = [0.01 * math.cos(0.8 * 0.01 * (k + 1)) for k in range(case["steps"])]
    else:  # ground: from the MP2 guess
        s["t2"] = _mp2(d["tei"], d["fock"], case["o"]).to(torch.complex128).contiguous()
        s["t1"] = torch.zeros((case["o"], case["v"]), dtype=torch.complex128, device="cuda")
    run(s)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "rhs":
        return s["eng"].rhs(c["method"], BLOCKS.index(c["block"]), *s["state"], F=s["F"])
    if kind == "step":
        state, mu = s["eng"].rk4_step(c["method"], s["state"], 0.0, 0.005, s["field"])
        return list(state) + [mu]
    if kind == "propagate":
        state, mu = s["eng"].propagate(c["method"], s["state"], 0.0, 0.005, c["steps"], s["field"])
        return list(state) + [mu]
    if kind == "gradient":
        J, gE, a = adjoint(s["eng"], c["method"], s["state"], 0.0, 0.01, c["steps"], s["weights"], field=s["field"],
                           want_state_grad=True)
        return [J, gE] + list(a)
    if kind == "ground":
        E, it, t1, t2 = s["eng"].ground_state(c["method"], 0, s["t1"], s["t2"], maxsize=8, maxiter=c["iters"], E_min=0.0)
        return [E, it, t1, t2]
    if kind == "spectrum":
        return list(spectrum(s["mu"], 0.005))
    return tei_from_df_device(s["B"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _rhs_flops(method, block, o, v):
    """Leading contractions of one residual and one trajectory, re-associated so that no v^4
    intermediate is formed (4 flops a real-complex multiply-add, 8 a complex one)."""
    if block == "T1":
        return 4 * (2 * o**2 * v**3 + 2 * o**3 * v**2 + o * v**3)
    if method == "CCSD":
        if block == "T2":
            return 8 * o**2 * v**4 + 24 * o**3 * v**3 + 28 * o**4 * v**2
        if block == "L1":
            return 4 * o * v**4 + 4 * o**2 * v**4 + 12 * o**3 * v**3 + 16 * o**2 * v**3
        return 4 * o**2 * v**4 + 20 * o**3 * v**3 + 24 * o**4 * v**2
    if block == "T2":
        return 4 * o**2 * v**4 + 4 * o**3 * v**3 + 20 * o**4 * v**2
    if block == "L1":
        return 4 * o * v**4 + 4 * o**3 * v**3 + 16 * o**2 * v**3
    return 8 * o**2 * v**3 + 16 * o**3 * v**2


def _tei_bytes(block, o, v):
    """The integral blocks a residual reads, each class of permutations once."""
    n = o**4 + o**3 * v + 2 * o**2 * v**2 + o * v**3 + (0 if block == "T1" else v**4)
    return 8 * (n if block != "T1" else n - o**4)


def work(case):
    kind = case["kind"]
    if kind == "spectrum":
        n = case["steps"]
        return {"bytes": 48 * n, "flops": 10 * n * max(1.0, math.log2(n))}
    o, v, nb = case["o"], case["v"], case.get("nb", 1)
    if kind == "integrals":
        n = o + v
        return {"bytes": 8 * n**4 + 8 * case["nq"] * n * n, "flops": 2 * case["nq"] * n**4}
    amps = 16 * (o * v + (o * v) ** 2)  # one (singles, doubles) pair
    full = sum(_rhs_flops(case["method"], b, o, v) for b in BLOCKS)
    if kind == "rhs":
        b = case["block"]
        out = 16 * (o * v if b in ("T1", "L1") else (o * v) ** 2)
        ins = amps * (1 if b[0] == "T" else 2) + 16 * (o + v) ** 2
        return {"bytes": _tei_bytes(b, o, v) + nb * (ins + out), "flops": nb * _rhs_flops(case["method"], b, o, v)}
    steps = case.get("steps", 1)
    if kind == "ground":
        t = _rhs_flops(case["method"], "T1", o, v) + _rhs_flops(case["method"], "T2", o, v)
        sweeps = 9 + case["iters"] - 1
        return {"bytes": _tei_bytes("T2", o, v) + sweeps * 3 * amps, "flops": sweeps * t}
    # the parts that the frozen amplitudes fix are done once a step: about half of four stages
    w = {"bytes": _tei_bytes("T2", o, v) + steps * nb * 4 * amps, "flops": steps * nb * 2.5 * full}
    if kind == "gradient":
        w["flops"] *= 3.0
    return w


# ---------------------------------------------------------------------------
# the equations in plain torch, complex128 (index strings and prefactors are the method's)
# ---------------------------------------------------------------------------
def _outer(x, y):
    return x[:, None, :, None] * y[None, :, None, :]


def _pij(x):
    return x - x.transpose(0, 1)


def _pab(x):
    return x - x.transpose(2, 3)


def _pijab(x):
    return _pij(_pab(x))


class _Plain:
    def __init__(self, tei, o, mu):
        self.g, self.o, self.mu, self._blk = tei, o, mu, {}

    def G(self, b):
        if b not in self._blk:
            o = self.o
            s = tuple(slice(0, o) if c == "o" else slice(o, None) for c in b)
            self._blk[b] = self.g[s].to(torch.complex128)
        return self._blk[b]

    def fb(self, F, b):
        o = self.o
        s = tuple(slice(0, o) if c == "o" else slice(o, None) for c in b)
        return F[s]

    e = staticmethod(torch.einsum)

    def fme(self, t1, F):
        return self.fb(F, "ov") + self.e("mnef,nf->me", self.G("oovv"), t1)

    def fae_fmi(self, t1, t2, F):
        e, G = self.e, self.G
        tau = t2 + _outer(t1, t1)
        fae = (self.fb(F, "vv") - 0.5 * e("me,ma->ae", self.fb(F, "ov"), t1) + e("mafe,mf->ae", G("ovvv"), t1)
               - 0.5 * e("mnef,mnaf->ae", G("oovv"), tau))
        fmi = (self.fb(F, "oo") + 0.5 * e("me,ie->mi", self.fb(F, "ov"), t1) + e("mnie,ne->mi", G("ooov"), t1)
               + 0.5 * e("mnef,inef->mi", G("oovv"), tau))
        return fae, fmi

    def T1(self, method, t1, t2, l1, l2, F):
        e, G = self.e, self.G
        fae, fmi = self.fae_fmi(t1, t2, F)
        return (self.fb(F, "ov") + e("ae,ie->ia", fae, t1) - e("mi,ma->ia", fmi, t1) + e("me,imae->ia", self.fme(t1, F), t2)
                - e("naif,nf->ia", G("ovov"), t1) - 0.5 * e("nmei,mnae->ia", G("oovo"), t2)
                - 0.5 * e("maef,imef->ia", G("ovvv"), t2))

    def T2(self, method, t1, t2, l1, l2, F):
        e, G = self.e, self.G
        tt = _outer(t1, t1)
        tau = tt - tt.transpose(2, 3)
        wmn2 = G("oooo") + _pab(e("mnie,je->mnij", G("ooov"), t1)) + 0.25 * _pab(e("mnef,ijef->mnij", G("oovv"), tt))
        wab = G("vvvv") - _pij(e("amef,mb->abef", G("vovv"), t1))
        wab2 = wab + 0.25 * e("mnef,mnab->abef", G("oovv"), tau)
        r = (G("oovv") + 0.5 * e("mnij,mnab->ijab", wmn2, tau) + 0.5 * e("abef,ijef->ijab", wab2, tau)
             + _pij(e("abej,ie->ijab", G("vvvo"), t1)) - _pab(e("mbij,ma->ijab", G("ovoo"), t1)))
        tring = e("mbij,ma->ijab", e("mbej,ie->mbij", G("ovvo"), t1), t1)
        if method == "CC2":
            return (r + _pab(e("be,ijae->ijab", self.fb(F, "vv"), t2)) - _pij(e("mj,imab->ijab", self.fb(F, "oo"), t2))
                    - _pijab(tring))
        fae, fmi = self.fae_fmi(t1, t2, F)
        fme = self.fme(t1, F)
        be = fae - 0.5 * e("me,mb->be", fme, t1)
        mj = fmi + 0.5 * e("me,je->mj", fme, t1)
        wmn = (G("oooo") + _pab(e("mnie,je->mnij", G("ooov"), t1))
               + e("mnef,ijef->mnij", G("oovv"), 0.25 * t2 + 0.5 * tau))
        wabt = wab + e("mnef,mnab->abef", G("oovv"), 0.25 * t2 + 0.5 * tau)
        wmb = (G("ovvo") - e("mnej,nb->mbej", G("oovo"), t1) - e("mnef,jnfb->mbej", G("oovv"), 0.5 * t2 + tt)
               + e("mbef,jf->mbej", G("ovvv"), t1))
        return (r + _pab(e("be,ijae->ijab", be, t2)) - _pij(e("mj,imab->ijab", mj, t2))
                + 0.5 * e("mnij,mnab->ijab", wmn, t2) + 0.5 * e("abef,ijef->ijab", wabt, t2)
                + _pijab(e("mbej,imae->ijab", wmb, t2) - tring))

    def lr(self, t1, t2, F):
        e, G = self.e, self.G
        tau = 0.5 * t2 + _outer(t1, t1)
        fea = (self.fb(F, "vv") - e("ma,me->ea", self.fb(F, "ov"), t1) + e("emaf,mf->ea", G("vovv"), t1)
               - e("mnaf,mnef->ea", G("oovv"), tau))
        fim = (self.fb(F, "oo") + e("ie,me->im", self.fb(F, "ov"), t1) + e("inmf,nf->im", G("ooov"), t1)
               + e("inef,mnef->im", G("oovv"), tau))
        return fea, fim

    def lam_common(self, t1, t2):
        e, G = self.e, self.G
        tt = _outer(t1, t1)
        wie = (G("ovvo") + e("eifa,mf->ieam", G("vovv"), t1) - e("nima,ne->ieam", G("ooov"), t1)
               - e("ijab,mjbe->ieam", G("oovv"), t2 + tt))
        tq = 0.25 * t2 + 0.5 * tt
        wmn = 0.5 * G("oooo") + e("ijme,ne->ijmn", G("ooov"), t1) + e("ijfe,mnfe->ijmn", G("oovv"), tq)
        wab = 0.5 * G("vvvv") - e("emab,mf->efab", G("vovv"), t1) + e("nmab,nmef->efab", G("oovv"), tq)
        return wie, wmn, wab, tq

    def wfiea(self, t1):
        return self.G("vovv") - self.e("jiea,jf->fiea", self.G("oovv"), t1)

    def wmina(self, t1):
        return self.G("ooov") + self.e("mifa,nf->mina", self.G("oovv"), t1)

    def L1(self, method, t1, t2, l1, l2, F):
        e, G = self.e, self.G
        fea, fim = self.lr(t1, t2, F)
        fme = self.fme(t1, F)
        r = fme + e("ea,ie->ia", fea, l1) - e("im,ma->ia", fim, l1)
        tt = _outer(t1, t1)
        if method == "CC2":
            base = G("ovvo") + e("mbef,jf->mbej", G("ovvv"), t1)
            x = e("mnej,nb->mbej", G("oovo"), t1) + e("mnef,jnfb->mbej", G("oovv"), tt)
            r = r - e("ijab,bj->ia", G("oovv"), e("me,mjbe->bj", l1, t2)) + e("ieam,me->ia", base - x, l1)
            tau = tt - tt.transpose(2, 3)
            wmn = G("oooo") + _pab(e("mnie,je->mnij", G("ooov"), t1)) - 0.5 * e("ijef,mnfe->ijmn", G("oovv"), tau)
            wmb = (G("ovoo") - e("nb,mnij->mbij", t1, wmn) + 0.5 * e("mbef,ijef->mbij", G("ovvv"), tau)
                   - e("mbei,je->mbij", G("ovvo"), t1) + e("mbej,ie->mbij", G("ovvo"), t1))
            z = base - 0.5 * x
            wab = (G("vvvo") + e("abef,if->abei", G("vvvv"), t1) + e("maei,mb->abei", z, t1) - e("mbei,ma->abei", z, t1))
            return r - 0.5 * e("iemn,mnae->ia", wmb, l2) + 0.5 * e("efam,imef->ia", wab, l2)
        wie, wmn, wab, tq = self.lam_common(t1, t2)
        jf = -G("ovvo") + e("jnab,nmfb->jfam", G("oovv"), t2)
        wef = (0.5 * G("vvvo") + 0.5 * e("na,mnef->efam", fme, t2) + e("efab,mb->efam", wab, t1) + e("jfam,je->efam", jf, t1)
               + e("jnam,jnef->efam", G("oovo"), tq) - e("jfab,jmeb->efam", G("ovvv"), t2))
        ib = -G("ovvo") - e("inef,nmfb->ibem", G("oovv"), t2)
        wib = (-0.5 * G("ovoo") + 0.5 * e("ie,jmbe->ibjm", fme, t2) + e("injm,nb->ibjm", wmn, t1) + e("ibem,je->ibjm", ib, t1)
               - e("ibef,jmef->ibjm", G("ovvv"), tq) + e("inem,jneb->ibjm", G("oovo"), t2))
        gfe = -0.5 * e("mnfb,mneb->fe", l2, t2)
        gmn = 0.5 * e("njed,mjed->nm", l2, t2)
        return (r + e("ieam,me->ia", wie, l1) + e("efam,imef->ia", wef, l2) + e("ibjm,jmab->ia", wib, l2)
                - e("fe,fiea->ia", gfe, self.wfiea(t1)) - e("nm,mina->ia", gmn, self.wmina(t1)))

    def L2(self, method, t1, t2, l1, l2, F):
        e, G = self.e, self.G
        fme = self.fme(t1, F)
        r = G("oovv") + _pij(e("ejab,ie->ijab", self.wfiea(t1), l1)) - _pab(e("ijmb,ma->ijab", self.wmina(t1), l1))
        lf = _outer(l1, fme)
        if method == "CC2":  # the method sums e over F_vv alone in this term
            x = l2 * self.fb(F, "vv").sum(0)
            return r + _pab(x) - _pij(e("imab,jm->ijab", l2, self.fb(F, "oo"))) + _pijab(lf)
        fea, fim = self.lr(t1, t2, F)
        wie, wmn, wab, _ = self.lam_common(t1, t2)
        gfe = -0.5 * e("mnfb,mneb->fe", l2, t2)
        gmn = 0.5 * e("njed,mjed->nm", l2, t2)
        return (r + _pab(e("eb,ijae->ijab", fea, l2) + e("ijfb,af->ijab", G("oovv"), gfe))
                - _pij(e("jm,imab->ijab", fim, l2) + e("mjab,im->ijab", G("oovv"), gmn))
                + e("ijmn,mnab->ijab", wmn, l2) + e("efab,ijef->ijab", wab, l2)
                + _pijab(e("jebm,imae->ijab", wie, l2) + lf))

    def dipole(self, t1, t2, l1, l2):
        e = self.e
        ll, vv = e("mnef,inef->mi", l2, t2), e("mnef,mnaf->ea", l2, t2)
        dij = -e("je,ie->ij", l1, t1) - 0.5 * e("jmea,imea->ij", l2, t2)
        dab = e("nb,na->ab", l1, t1) + 0.5 * e("mneb,mnea->ab", l2, t2)
        dai = (t1.T + e("me,miea->ai", l1, t2) - e("ae,ie->ai", e("me,ma->ae", l1, t1), t1) - 0.5 * e("ea,ie->ai", vv, t1)
               - 0.5 * e("mi,ma->ai", ll, t1))
        rho = torch.cat([torch.cat([dij, l1], 1), torch.cat([dai, dab], 1)], 0)
        return torch.stack([(m * rho).sum() for m in self.mu])

    def step(self, method, state, E, dt, fock, mu, rounded=True):
        """One step of the loop body; E: the field at the four stages."""
        new = []
        for b, name in enumerate(BLOCKS):
            f, k, acc = getattr(self, name), None, 0.0
            for s, (h, w) in enumerate(((0.0, 1.0), (dt / 2, 2.0), (dt / 2, 2.0), (dt, 1.0))):
                y = list(state)
                if s:
                    y[b] = state[b] + h * k
                k = f(method, *y, fock - E[s] * mu)
                acc = acc + w * k
            old = state[b]
            if rounded:
                old = torch.view_as_complex(torch.round(torch.view_as_real(old) * 1e15) / 1e15)
            new.append(old + (-1j if b < 2 else 1j) * (dt / 6.0) * acc)
        return new


def _stage_fields(A, w0, dt, steps):
    t, out = 0.0, []
    for _ in range(steps):
        t += dt
        out.append([A * math.sin(w0 * x) for x in (t, t + dt / 2, t + dt / 2, t + dt)])
    return out


def _exact_ground(case, d, p):
    o, dev = case["o"], d["fock"].device
    F = d["fock"].to(torch.complex128)
    eps = torch.diagonal(d["fock"])
    d1 = eps[:o, None] - eps[None, o:]
    d2 = d1[:, None, :, None] + d1[None, :, None, :]
    x = [torch.zeros((o, case["v"]), dtype=torch.complex128, device=dev), _mp2(d["tei"], d["fock"], o).to(torch.complex128)]

    def sweep(x):
        return [x[0] + p.T1(case["method"], *x, None, None, F) / d1, x[1] + p.T2(case["method"], *x, None, None, F) / d2]

    def energy(x):
        g = p.G("oovv")
        return float(((p.fb(F, "ov") * x[0]).sum() + 0.25 * (g * x[1]).sum() + 0.5 * (g * _outer(x[0], x[0])).sum()).real)

    size = 8
    x = sweep(x)
    store, err = [x], []
    for _ in range(size):
        x = sweep(x)
        store.append(x)
        err.append([a - b for a, b in zip(store[-1], store[-2])])
    E, it = 0.0, 0
    for _ in range(1, case["iters"]):
        B = -np.ones((size + 1, size + 1))
        B[-1, -1] = 0.0
        for a in range(size):
            for b in range(size):
                B[a, b] = float(sum((u * w).sum() for u, w in zip(err[a], err[b])).real)
        rhs = np.zeros(size + 1)
        rhs[-1] = -1.0
        c = np.linalg.solve(B, rhs)
        old = [sum(c[a] * store[a + 1][k] for a in range(size)) for k in range(2)]
        E, it = energy(old), it + 1
        x = sweep(old)
        store = store[1:] + [x]
        err = err[1:] + [[a - b for a, b in zip(x, old)]]
    return [E, it, x[0], x[1]]


def exact(case, seed):
    kind = case["kind"]
    if kind == "spectrum":
        mu = prepare(case, seed)["mu"].cpu().numpy()
        n = len(mu)
        k = np.arange(n) - n // 2
        return [k / (n * 0.005) * (2.0 * np.pi) * 27.211, np.fft.fftshift(np.fft.fft(mu.real)),
                np.fft.fftshift(np.fft.fft(mu.imag))]
    d = _inputs(case, seed)
    if kind == "integrals":
        return _tei(d["B"])
    p = _Plain(d["tei"], case["o"], d["mu"])
    if kind == "ground":
        return _exact_ground(case, d, p)
    nb, method = case["nb"], case["method"]
    states = [[x if nb == 1 else x[b] for x in d["state"]] for b in range(nb)]
    if kind == "rhs":
        F = _dressed(case, d)
        r = [getattr(p, case["block"])(method, *st, F if nb == 1 else F[b]) for b, st in enumerate(states)]
        return r[0] if nb == 1 else torch.stack(r)
    steps, fock = case.get("steps", 1), d["fock"].to(torch.complex128)
    if kind == "gradient":
        st = [x.clone().requires_grad_(True) for x in states[0]]
        E = torch.tensor(_stage_fields(A0, W0, 0.01, steps), dtype=torch.complex128, device=fock.device, requires_grad=True)
        y, J = st, 0.0
        for n in range(steps):
            y = p.step(method, y, E[n], 0.01, fock, d["mu"][2], rounded=False)
            J = J + 0.01 * math.cos(0.8 * 0.01 * (n + 1)) * p.dipole(*y)[2].real
        g = torch.autograd.grad(J, [E] + st)
        return [J.detach().reshape(1), g[0].conj().resolve_conj().reshape(steps, 4, 1)] + [x.conj().resolve_conj() for x in g[1:]]
    f = _fields(case) if nb > 1 else [(2, A0, W0)]
    ends, mus = [], []
    for b, st in enumerate(states):
        pol, A, w = f[b]
        tr = []
        for E in _stage_fields(A, w, 0.005, steps):
            st = p.step(method, st, E, 0.005, fock, d["mu"][pol])
            tr.append(p.dipole(*st))
        ends.append(st)
        mus.append(torch.stack(tr))  # [step][component]
    out = [x if nb == 1 else torch.stack([e[k] for e in ends]) for k, x in enumerate(ends[0])]
    if kind == "step":
        out.append(mus[0][0] if nb == 1 else torch.stack([m[0] for m in mus]))
    else:
        tr = [m[:, f[b][0]] for b, m in enumerate(mus)]
        out.append(tr[0] if nb == 1 else torch.stack(tr, 1))
    return out
