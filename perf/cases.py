"""The work that users of this package have it do, as timed cases.

A case names a system (He n=2, H2 n=3, LiH n=5), a basis size K and one of the
package's public calls (``call``):

  host       Engine.outprod: host x in, host (f, g) out -- what a SciPy optimiser
             or a C / Fortran driver calls once per line-search step
  dropin     outprod.outprod: the reference's objective with its module state,
             H and S copied back into ``shared``
  device     Engine.outprod_device: x, f and g stay on the GPU (restartable
             optimisers, the benchmark's headline)
  autograd   autograd.energy forward and backward, gradients with respect to iv, C
  matrices   Engine.build_matrices: H, S, Kinetic, Potential and [E, norm], the
             start and the end of every driver run
  dipole     Engine.dipole: the end of every driver run (nst^2 terms per pair)
  terms      Engine.matel and Engine.gradel of a list of (stf, ii, jj) terms
  batch      BatchEngine plan + step over many bases of the three systems, what
             the serving loop launches for the requests that are ready

Engines are set up as the drop-in module and the benchmark set theirs up, with
the autotuner's setting for their (n, nst, K).  Parameters follow the
distributions of ``synth`` (L_k diagonal uniform, off-diagonal normal(0, 0.3),
shifts normal(0, 0.05)); C has random signs, as an eigenvector of the
generalised problem has.
"""
import math

import numpy as np
import torch

from nbo_correlatedgaussians_b200 import autotune, shared, synth
from nbo_correlatedgaussians_b200.autograd import energy
from nbo_correlatedgaussians_b200.batch import BatchEngine
from nbo_correlatedgaussians_b200.engine import Engine
from nbo_correlatedgaussians_b200.outprod import outprod as dropin_outprod
from nbo_correlatedgaussians_b200.problem import Problem

NST = {"He": 2, "H2": 4, "LiH": 24}
N = {"He": 2, "H2": 3, "LiH": 5}


def listed():
    return [
        # the smallest basis in use (the reference's own input has K = 12): latency of one optimiser step
        {"name": "lih_k12_host", "call": "host", "system": "LiH", "K": 12},
        # a working basis through the drop-in objective, with H and S copied back as the reference has them
        {"name": "lih_k96_dropin", "call": "dropin", "system": "LiH", "K": 96},
        # ragged sizes of the small systems, one optimiser step each
        {"name": "he_k331_host", "call": "host", "system": "He", "K": 331},
        {"name": "h2_k157_host", "call": "host", "system": "H2", "K": 157},
        # the largest bases of the small systems (He: the largest run of the serving stream)
        {"name": "he_k2032_device", "call": "device", "system": "He", "K": 2032},
        {"name": "h2_k2048_device", "call": "device", "system": "H2", "K": 2048},
        # the benchmark's headline evaluation
        {"name": "lih_k1024_device", "call": "device", "system": "LiH", "K": 1024},
        # E and its gradient through torch.autograd
        {"name": "h2_k2048_autograd", "call": "autograd", "system": "H2", "K": 2048},
        # the driver's matrix build and its dipole
        {"name": "lih_k301_matrices", "call": "matrices", "system": "LiH", "K": 301},
        {"name": "lih_k160_dipole", "call": "dipole", "system": "LiH", "K": 160},
        # tables of single elements and of single element gradients
        {"name": "lih_terms_2000", "call": "terms", "system": "LiH", "K": 128, "terms": 2000},
        # one step of the batched / serving path over bases of all three systems
        {"name": "mixed_batch_24", "call": "batch", "he": 6, "h2": 9, "lih": 9, "lo": 48, "hi": 1000},
    ]


# largest K drawn per call and system: a drawn case costs no more than the largest listed one
DRAW_MAX = {"host": {"He": 2048, "H2": 2048, "LiH": 1000}, "dropin": {"He": 1024, "H2": 1024, "LiH": 700},
            "device": {"He": 2048, "H2": 2048, "LiH": 1000}, "autograd": {"He": 2048, "H2": 2048, "LiH": 500},
            "matrices": {"He": 2048, "H2": 2048, "LiH": 700}, "dipole": {"He": 1000, "H2": 700, "LiH": 160},
            "terms": {"He": 512, "H2": 512, "LiH": 512}}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["host", "host", "dropin", "device", "device", "autograd", "matrices", "dipole", "terms",
                       "batch"])
    if call == "batch":
        lo = _log_int(rng, 24, 96)
        return {"call": call, "he": rng.randint(0, 8), "h2": rng.randint(1, 8), "lih": rng.randint(1, 8), "lo": lo,
                "hi": _log_int(rng, 2 * lo, 700)}
    system = rng.choice(["He", "H2", "LiH"])
    case = {"call": call, "system": system, "K": _log_int(rng, 12, DRAW_MAX[call][system])}
    if call == "terms":
        case["terms"] = _log_int(rng, 1, 4000)
    return case


# ---------------------------------------------------------------- inputs
def _problem(system, K, seed):
    p = synth.make_problem(system, K, seed)
    p.C = np.random.default_rng([seed, K]).normal(size=K) / math.sqrt(K)
    return p


def _problems(case, seed):
    """The bases of a case, from its seed alone (sizes from the case alone)."""
    if case["call"] != "batch":
        return [_problem(case["system"], case["K"], seed)]
    sizes = np.random.default_rng(case["lo"] * 1000 + case["hi"])
    out = []
    for system, count in (("He", case["he"]), ("H2", case["h2"]), ("LiH", case["lih"])):
        for i in range(count):
            hi = min(case["hi"], 512) if system == "He" else case["hi"]
            out.append(_problem(system, synth.log_uniform_int(sizes, case["lo"], hi), seed + 7919 * (len(out) + 1)))
    return out


def _terms(case, seed):
    rng = np.random.default_rng([seed, case["terms"]])
    c = case["terms"]
    return np.stack([rng.integers(1, NST[case["system"]] + 1, c), rng.integers(1, case["K"] + 1, c),
                     rng.integers(1, case["K"] + 1, c)], 1).astype(np.int32)


_settings = {}  # the autotuner's settings, found once per process as a user's program finds them


def _tuned(eng, x, K):
    key = (eng.n, eng.nst, K.bit_length())
    if key in _settings:
        autotune.apply(eng, _settings[key])
    else:
        _settings[key] = autotune.tuned(eng, x, K)


def prepare(case, seed):
    call = case["call"]
    probs = _problems(case, seed)
    if call == "batch":
        be = BatchEngine(probs, tune=False)
        for eng, x, p in zip(be.engines, be.x, probs):
            _tuned(eng, x, p.K)
        return {"call": call, "engine": be}
    p = probs[0]
    if call == "dropin":
        sh = shared
        sh.M, sh.ne, sh.nst, sh.efs, sh.svh, sh.skp, sh.siv = p.K, p.n, p.nst, p.efs, p.svh, p.skp, p.siv
        sh.mass, sh.ncv, sh.scvv, sh.iv, sh.C = p.mass, p.ncv, p.scvv, p.iv.copy(), p.C.copy()
        sh.sml = np.ascontiguousarray(np.transpose(p.sml, (1, 2, 0)))
        sh.sms = np.ascontiguousarray(np.transpose(p.sms, (1, 2, 0)))
        sh.H, sh.S = np.zeros((p.K, p.K)), np.zeros((p.K, p.K))
        sh.grad = np.zeros(p.siv + p.K)
        return {"call": call, "x": p.x}
    eng = Engine(p)
    st = {"call": call, "engine": eng, "K": p.K}
    x = torch.from_numpy(p.x).to(eng.device)
    _tuned(eng, x, p.K)
    if call == "host":
        st["x"] = p.x
    elif call == "device":
        st["x"], st["g"], st["f"] = x, torch.empty_like(x), torch.empty(1, dtype=torch.float64, device=x.device)
    elif call == "autograd":
        st["iv"] = x[:p.siv].clone().requires_grad_(True)
        st["C"] = x[p.siv:].clone().requires_grad_(True)
    else:
        st["iv"], st["C"] = x[:p.siv].clone(), x[p.siv:].clone()
        if call == "terms":
            st["terms"] = _terms(case, seed)
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    call = st["call"]
    if call == "batch":
        be = st["engine"]
        be.plan()
        be.step()
        return {"f": be.f, "g": be.g}
    if call == "dropin":
        f, g = dropin_outprod(st["x"])
        return {"f": np.float64(f), "g": g, "H": shared.H, "S": shared.S}
    eng = st["engine"]
    if call == "host":
        f, g = eng.outprod(st["x"])
        return {"f": np.float64(f), "g": g}
    if call == "device":
        f, g = eng.outprod_device(st["x"], st["K"], g=st["g"], f=st["f"])
        return {"f": f, "g": g}
    if call == "autograd":
        E = energy(st["iv"], st["C"], eng)
        gi, gc = torch.autograd.grad(E, (st["iv"], st["C"]))
        return {"f": E.detach(), "giv": gi, "gC": gc}
    if call == "matrices":
        H, S, Kin, Pot, en = eng.build_matrices(st["iv"], st["C"], K=st["K"])
        return {"H": H, "S": S, "Kin": Kin, "Pot": Pot, "en": en}
    if call == "dipole":
        comps, dip = eng.dipole(st["iv"], st["C"])
        return {"comps": comps, "dip": dip}
    mat = eng.matel(st["iv"], st["terms"], K=st["K"])
    tg, tgs = eng.gradel(st["iv"], st["terms"], K=st["K"])
    return {"mat": mat, "tg": tg, "tgs": tgs}


# ---------------------------------------------------------------- what a pass cannot do without
def _term_flops(n, grad):
    """FP64 operations of one (k, l, P) term in n-space (FMA = 2, a root, quotient
    or exponential = 1): B = A_k + A_l', its inverse and determinant, T = B^-1 e,
    the overlap, the kinetic trace and the n(n+1)/2 Coulomb terms; with the
    gradient, their derivatives with respect to B and e and the weighted sums
    of the H and S parts for bra and ket."""
    t, v = n * (n + 1) // 2, 3 * n
    f = (t + n * n * n + n) + (v + 6 * n * n) + (2 * v + 12) + (8 * t + 2 * t + 2 * v) + 36 * t
    if grad:
        f += 36 * t + 2 * (n * n * n + n * t) + 12 * n * n + 12 * t + 6 * t + 8 * (t + v)
    return f


def work(case):
    call = case["call"]
    n_bytes = flops = 0
    for p in ([(N[s], NST[s], case["K"]) for s in [case["system"]]] if call != "batch"
              else [(p.n, p.nst, p.K) for p in _problems(case, 0)]):
        n, nst, K = p
        blk = n * (n + 1) // 2 + 3 * n
        x = 8 * K * (blk + 1)
        pairs = K * (K + 1) // 2
        if call == "matrices":
            n_bytes, flops = n_bytes + x + 32 * K * K, flops + pairs * nst * _term_flops(n, False)
        elif call == "dipole":
            # the operator is linear in the position and the terms form a group: nst distinct overlaps per pair
            n_bytes, flops = n_bytes + x + 24 * (n + 1), flops + pairs * nst * (_term_flops(n, False) - 46 * n * (n + 1) // 2)
        elif call == "terms":
            c = case["terms"]
            n_bytes += x + c * (12 + 32 + 16 * blk)
            flops += c * (_term_flops(n, False) + _term_flops(n, True))
        else:
            n_bytes += 2 * x + 8 + (16 * K * K if call == "dropin" else 0)
            flops += pairs * nst * _term_flops(n, True)
    return {"bytes": n_bytes, "flops": flops}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
PADE_NUM = [1.0, 0.213271302, 0.062934446, 0.00769838037, 0.000758433197, 0.0000564691197]
PADE_DEN = [1.0, 0.879937801, 0.338450368, 0.0738522953, 0.0101431553, 0.000955528842, 0.000072026652]
SPLIT = 16.3578


def _poly(c, z):
    v = torch.full_like(z, c[-1])
    for a in reversed(c[:-1]):
        v = v * z + a
    return v


def _f0(z):
    """The reference's Pade form of the Boys function below z = 16.3578, sqrt(pi / 4z) above."""
    small = z <= SPLIT
    zs = torch.where(small, z, torch.ones_like(z))
    zl = torch.where(small, torch.full_like(z, 20.0), z)
    return torch.where(small, torch.sqrt(_poly(PADE_NUM, zs) / _poly(PADE_DEN, zs)), torch.sqrt(math.pi / (4.0 * zl)))


class _Plain:
    """Matrix elements of one problem from the formulas, in n-space."""

    def __init__(self, p: Problem, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.n, self.K, self.nst, self.efs, self.dev = p.n, p.K, p.nst, p.efs, dev
        self.M, self.q, self.w, self.sml, self.sms = t(p.mass), t(p.ncv), t(p.scvv), t(p.sml), t(p.sms)
        v = torch.zeros((p.n * (p.n + 1) // 2, p.n), dtype=torch.float64, device=dev)
        c = torch.zeros(p.n * (p.n + 1) // 2, dtype=torch.float64, device=dev)
        i = 0
        for b in range(1, p.n + 1):
            for a in range(b):
                v[i, b - 1] = 1.0
                if a:
                    v[i, a - 1] = -1.0
                c[i] = 2.0 * p.ncv[a] * p.ncv[b] / math.sqrt(math.pi)
                i += 1
        self.v, self.c = v, c
        lo = [(r, col) for col in range(p.n) for r in range(col, p.n)]
        self.lr, self.lc = torch.tensor([r for r, _ in lo], device=dev), torch.tensor([c_ for _, c_ in lo], device=dev)

    def basis(self, iv):
        """L (K, n, n) and s (K, n, 3) of the packed parameters."""
        b = iv.reshape(-1, self.n * (self.n + 1) // 2 + 3 * self.n)
        L = torch.zeros((b.shape[0], self.n, self.n), dtype=torch.float64, device=self.dev)
        L = L.index_put((torch.arange(b.shape[0], device=self.dev)[:, None], self.lr[None], self.lc[None]), b[:, :self.lr.numel()])
        return L, b[:, self.lr.numel():].reshape(-1, self.n, 3)

    def mapped(self, L, s, P):
        """A and s of a basis after symmetry term(s) P (an index, or one per function)."""
        A = L @ L.transpose(-1, -2)
        m = self.sml[P]
        m = m.transpose(-1, -2)
        return m @ A @ self.sml[P], (self.sms[P] @ s.reshape(-1, 3 * self.n, 1)).reshape(-1, self.n, 3)

    def core(self, Ak, sk, dk, Al, sl, dl):
        """B^-1, T and the overlap; d*: |L| of each function."""
        B = Ak + Al
        e = Ak @ sk + Al @ sl
        Bi = torch.linalg.inv(B)
        T = Bi @ e
        ex = (e * T).sum((-1, -2)) - (sk * (Ak @ sk)).sum((-1, -2)) - (sl * (Al @ sl)).sum((-1, -2))
        ov = 8.0 ** (0.5 * self.n) * (dk * dl / torch.linalg.det(B)) ** 1.5 * torch.exp(ex)
        return Bi, T, ov

    def elements(self, Ak, sk, dk, Al, sl, dl):
        """(ov, kinetic, Coulomb, Stark) of broadcast batches."""
        Bi, T, ov = self.core(Ak, sk, dk, Al, sl, dl)
        X = Ak @ Bi @ Al
        Y = Al @ (T - sl)
        tau = 3.0 * (self.M.T * X).sum((-1, -2)) - 2.0 * (Y * (self.M @ Y)).sum((-1, -2))
        Bv = Bi @ self.v.T                         # columns B^-1 v
        a = (self.v.T * Bv).sum(-2)
        b2 = ((self.v @ T) ** 2).sum(-1)
        rho = (self.c * _f0(b2 / a) / torch.sqrt(a)).sum(-1)
        sig = self.efs * (self.q[1:] * T[..., 2]).sum(-1)
        return ov, 2.0 * ov * tau, ov * rho, ov * sig


def _dets(L):
    return torch.diagonal(L, dim1=-2, dim2=-1).prod(-1).abs()


def _rows(pl, budget):
    """Row ranges whose (rows x kets) pairs stay within `budget` terms."""
    k = 0
    while k < pl.K:
        m = k + 1
        while m < pl.K and (m + 1 - k) * (m + 1) <= budget:
            m += 1
        yield k, m
        k = m


def _matrices(pl, iv, parts, budget=400_000):
    """H, S (and kinetic, potential) by lower-triangle rows, mirrored."""
    K = pl.K
    out = [torch.zeros((K, K), dtype=torch.float64, device=pl.dev) for _ in range(4 if parts else 2)]
    with torch.no_grad():
        L, s = pl.basis(iv)
        d, A = _dets(L), L @ L.transpose(-1, -2)
        for k0, k1 in _rows(pl, budget):
            for P in range(pl.nst):
                Al, sl = pl.mapped(L[:k1], s[:k1], P)
                ov, tk, er, zh = pl.elements(A[k0:k1, None], s[k0:k1, None], d[k0:k1, None], Al[None], sl[None], d[None, :k1])
                vals = [tk + er - zh, ov] + ([tk, er] if parts else [])
                for o, x in zip(out, vals):
                    o[k0:k1, :k1] += pl.w[P] * x
        return [torch.tril(o) + torch.tril(o, -1).T for o in out]


def _energy_gradient(p, dev):
    """E, dE/d[iv, C], H and S, the gradient by torch.autograd over rows of pairs."""
    pl = _Plain(p, dev)
    iv = torch.as_tensor(p.iv, dtype=torch.float64, device=dev)
    C = torch.as_tensor(p.C, dtype=torch.float64, device=dev)
    H, S = _matrices(pl, iv, False)
    cSc = C @ S @ C
    E = (C @ H @ C) / cSc
    gC = 2.0 * (H @ C - E * (S @ C)) / cSc
    iv = iv.requires_grad_(True)
    g = torch.zeros_like(iv)
    for k0, k1 in _rows(pl, 150_000):
        k = torch.arange(k0, k1, device=dev)[:, None]
        l = torch.arange(k1, device=dev)[None]
        wt = torch.where(l < k, 2.0, 1.0) * (l <= k) * C[k0:k1, None] * C[None, :k1]
        for P in range(pl.nst):
            L, s = pl.basis(iv[:k1 * p.blk])
            d = _dets(L)
            A = L @ L.transpose(-1, -2)
            Al, sl = pl.mapped(L, s, P)
            ov, tk, er, zh = pl.elements(A[k0:, None], s[k0:, None], d[k0:, None], Al[None], sl[None], d[None])
            part = (pl.w[P] * wt * (tk + er - zh - E * ov)).sum()
            g += torch.autograd.grad(part, iv)[0]
    return E, torch.cat([g / cSc, gC]), H, S


def _dipole(p, dev):
    pl = _Plain(p, dev)
    with torch.no_grad():
        L, s = pl.basis(torch.as_tensor(p.iv, dtype=torch.float64, device=dev))
        C = torch.as_tensor(p.C, dtype=torch.float64, device=dev)
        d = _dets(L)
        kk = torch.arange(p.K, device=dev)
        wt = torch.where(kk[None] < kk[:, None], 2.0, 1.0) * (kk[None] <= kk[:, None]) * C[:, None] * C[None]
        num, den = torch.zeros((p.n, 3), dtype=torch.float64, device=dev), 0.0
        kets = [pl.mapped(L, s, P) for P in range(p.nst)]
        step = max(1, 400_000 // p.K)
        for Pe in range(p.nst):
            for P in range(p.nst):
                for k0 in range(0, p.K, step):
                    r = slice(k0, k0 + step)
                    _, T, ov = pl.core(kets[Pe][0][r, None], kets[Pe][1][r, None], d[r, None], kets[P][0][None], kets[P][1][None], d[None])
                    wo = wt[r] * pl.w[Pe] * pl.w[P] * ov
                    den = den + wo.sum()
                    num = num + (wo[..., None, None] * T).sum((0, 1))
        comps = num / den
        return comps.reshape(-1), (pl.q[1:, None] * comps).sum(0)


def _single_terms(p, terms, dev):
    pl = _Plain(p, dev)
    t = torch.as_tensor(terms.astype(np.int64) - 1, device=dev)
    blocks = torch.as_tensor(p.iv, dtype=torch.float64, device=dev).reshape(p.K, -1)
    bra = blocks[t[:, 1]].clone().requires_grad_(True)
    Lk, sk = pl.basis(bra.reshape(-1))
    Ll, sl0 = pl.basis(blocks[t[:, 2]].reshape(-1))
    Al, sl = pl.mapped(Ll, sl0, t[:, 0])
    ov, tk, er, zh = pl.elements(Lk @ Lk.transpose(-1, -2), sk, _dets(Lk), Al, sl, _dets(Ll))
    twice = torch.where(t[:, 1] == t[:, 2], 2.0, 1.0)[:, None]
    tg = torch.autograd.grad((tk + er - zh).sum(), bra, retain_graph=True)[0] * twice
    tgs = torch.autograd.grad(ov.sum(), bra)[0] * twice
    return torch.stack([ov, tk, er, zh], 1).detach(), tg, tgs


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    call = case["call"]
    probs = _problems(case, seed)
    p = probs[0]
    if call == "batch":
        got = [_energy_gradient(q, dev)[:2] for q in probs]
        return {"f": [E.reshape(1) for E, _ in got], "g": [g for _, g in got]}
    if call == "matrices":
        pl = _Plain(p, dev)
        H, S, Kin, Pot = _matrices(pl, torch.as_tensor(p.iv, dtype=torch.float64, device=dev), True)
        C = torch.as_tensor(p.C, dtype=torch.float64, device=dev)
        cSc = C @ S @ C
        return {"H": H, "S": S, "Kin": Kin, "Pot": Pot, "en": torch.stack([(C @ H @ C) / cSc, 1.0 / cSc])}
    if call == "dipole":
        comps, dip = _dipole(p, dev)
        return {"comps": comps, "dip": dip}
    if call == "terms":
        mat, tg, tgs = _single_terms(p, _terms(case, seed), dev)
        return {"mat": mat, "tg": tg, "tgs": tgs}
    E, g, H, S = _energy_gradient(p, dev)
    if call == "autograd":
        return {"f": E, "giv": g[:p.siv], "gC": g[p.siv:]}
    out = {"f": E.reshape(1) if call == "device" else E, "g": g}
    if call == "dropin":
        out["H"], out["S"] = H, S
    return out
