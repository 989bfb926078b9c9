"""TEST INFRASTRUCTURE: matrix elements, energy and gradient of a small basis in
extended precision (numpy's 80-bit ``longdouble``), from the formulas of
python/matel.py and python/gradel.py in n-space.

The kinetic part is written with the smaller of tr(M A_k) and tr(M A_l') and the
gradients per pair with D_k = S_k - T and D_l = T - S_l', so that nothing cancels
between a tight and a diffuse function; its errors are those of 64-bit mantissas
(2048 times smaller than double's)."""
from __future__ import annotations

import numpy as np

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")
NUM = [1.0, 0.213271302, 0.0629344460, 0.00769838037, 0.000758433197, 0.0000564691197]
DEN = [1.0, 0.879937801, 0.338450368, 0.0738522953, 0.0101431553, 0.000955528842, 0.0000720266520]


def _poly(c, z):
    v = np.zeros_like(z) + LD(c[-1])
    for a in c[-2::-1]:
        v = v * z + LD(a)
    return v


def _f0(z):
    """F0 and its derivative: the Pade form below the branch point, sqrt(pi / 4 z) above."""
    small = z <= LD(16.3578)
    zs, zl = np.where(small, z, LD(1)), np.where(small, LD(20), z)
    n, d = _poly(NUM, zs), _poly(DEN, zs)
    dn, dd = _poly([i * c for i, c in enumerate(NUM)][1:], zs), _poly([i * c for i, c in enumerate(DEN)][1:], zs)
    f = np.sqrt(n / d)
    fa = np.sqrt(PI / 4 / zl)
    return np.where(small, f, fa), np.where(small, f * (dn / n - dd / d) / 2, -fa / (2 * zl))


def _inverse(B):
    """Inverse and determinant of symmetric positive definite matrices (Cholesky)."""
    n = B.shape[-1]
    L, W = np.zeros_like(B), np.zeros_like(B)
    for j in range(n):
        L[..., j, j] = np.sqrt(B[..., j, j] - (L[..., j, :j] ** 2).sum(-1))
        for i in range(j + 1, n):
            L[..., i, j] = (B[..., i, j] - (L[..., i, :j] * L[..., j, :j]).sum(-1)) / L[..., j, j]
    for j in range(n):
        W[..., j, j] = 1 / L[..., j, j]
        for i in range(j + 1, n):
            W[..., i, j] = -(L[..., i, j:i] * W[..., j:i, j]).sum(-1) / L[..., i, i]
    det = np.prod([L[..., j, j] for j in range(n)], axis=0) ** 2
    return np.einsum("...ki,...kj->...ij", W, W), det


def _t(x):
    return np.swapaxes(x, -1, -2)


def _sym(x, y):
    return x @ _t(y) + y @ _t(x)


class Extended:
    def __init__(self, p):
        self.p, self.n, self.K = p, p.n, p.K
        n, K = p.n, p.K
        t = lambda a: np.asarray(a).astype(LD)  # noqa: E731
        b = t(p.iv).reshape(K, -1)
        self.tri = n * (n + 1) // 2
        self.L = np.zeros((K, n, n), LD)
        i = 0
        for c in range(n):
            for r in range(c, n):
                self.L[:, r, c] = b[:, i]
                i += 1
        self.s = b[:, self.tri:].reshape(K, n, 3)
        self.A = self.L @ _t(self.L)
        self.M, self.q, self.C = t(p.mass), t(p.ncv), t(p.C)
        self.det = np.abs(np.prod([self.L[:, j, j] for j in range(n)], axis=0))

    def ket(self, P):
        """A_l', s_l' of every basis function in the frame of symmetry term P."""
        m = self.p.sml[P].astype(LD)
        return m.T @ self.A @ m, (self.p.sms[P].astype(LD) @ self.s.reshape(self.K, -1).T).T.reshape(self.K, self.n, 3)

    def pairs(self, Ak, sk, dk, Al, sl, dl):
        """Values and one-sided derivatives of the pairs (k, l) given as broadcast
        arrays: ov, tk, ert, zht, and d h / d(A_k, s_k), d h / d(A_l', s_l') and the
        same of ov, apart from the A^-1 terms (coefficients 0.75 h and 0.75 ov)."""
        n, M = self.n, self.M
        B, e = Ak + Al, Ak @ sk + Al @ sl
        Bi, det = _inverse(B)
        T = Bi @ e
        Dk, Dl = sk - T, T - sl
        ex = (e * T).sum((-1, -2)) - (sk * (Ak @ sk)).sum((-1, -2)) - (sl * (Al @ sl)).sum((-1, -2))
        ov = np.sqrt(LD(8.0) ** n) * (dk * dl / det) ** LD(1.5) * np.exp(ex)
        Nk, Nl = Ak @ M @ Ak, Al @ M @ Al
        tk_, tl_ = np.einsum("ij,...ji->...", M, Ak), np.einsum("ij,...ji->...", M, Al)
        dot = lambda x, y: (x * y).sum((-1, -2))  # noqa: E731
        loose_k = tk_ <= tl_
        tau = np.where(loose_k, 3 * (tk_ - dot(Nk, Bi)) - 2 * dot(Dk, Nk @ Dk), 3 * (tl_ - dot(Nl, Bi)) - 2 * dot(Dl, Nl @ Dl))
        Y = np.where(loose_k[..., None, None], Ak @ Dk, Al @ Dl)
        rho, Z, W = np.zeros_like(ov), np.zeros_like(T), np.zeros_like(Bi)
        for qq in range(1, n + 1):
            for pp in range(qq):
                v = np.zeros(n, LD)
                v[qq - 1] = 1
                if pp:
                    v[pp - 1] = -1
                a = (v @ Bi @ v[:, None])[..., 0]
                bv = (v[None] @ T)[..., 0, :]
                z = (bv ** 2).sum(-1) / a
                f, df = _f0(z)
                c = 2 * self.q[pp] * self.q[qq] / np.sqrt(PI)
                rho += c * f / np.sqrt(a)
                Z += (c * df * a ** LD(-1.5))[..., None, None] * v[:, None] * bv[..., None, :]
                W += (c * a ** LD(-1.5) * (z * df + f / 2))[..., None, None] * np.outer(v, v)
        efs = LD(self.p.efs)
        sig = efs * (self.q[1:] * T[..., 2]).sum(-1)
        Z[..., 2] -= efs / 2 * self.q[1:]
        Qk = Bi @ (Z - 4 * Al @ (M @ Y))
        Ql = Bi @ (Z + 4 * Ak @ (M @ Y))
        h = (2 * tau + rho - sig)[..., None, None]
        o = ov[..., None, None]
        one = np.ones_like(h)
        gk = lambda x, w: -x * (LD(1.5) * Bi + Dk @ _t(Dk)) + w * (Bi @ (6 * Nl + W) @ Bi + _sym(Qk, Dk))  # noqa: E731
        gl = lambda x, w: -x * (LD(1.5) * Bi + Dl @ _t(Dl)) + w * (Bi @ (6 * Nk + W) @ Bi - _sym(Ql, Dl))  # noqa: E731
        bra = [(o * gk(h, one), o * (2 * Ak @ Qk - 2 * h * Y)), (o * gk(one, 0 * h), -2 * o * Y)]
        ket = [(o * gl(h, one), o * (2 * Al @ Ql + 2 * h * Y)), (o * gl(one, 0 * h), 2 * o * Y)]
        return ov, 2 * ov * tau, ov * rho, ov * sig, bra, ket

    def vech(self, G, D, L):
        """dF/d vech(L) from dF/dA = G + D A^-1."""
        gL = 2 * G @ L
        cols = []
        for c in range(self.n):
            for r in range(c, self.n):
                cols.append(gL[..., r, c] + (2 * D / L[..., c, c] if r == c else 0))
        return np.stack(cols, -1)

    def evaluate(self):
        """dict: E, g (GRADA blocks K x blk), gC, and H, S, T (kinetic) with aH, aT: the sums
        of the absolute values of their terms, which rounding errors are measured against."""
        p, K = self.p, self.K
        kk = np.arange(K)
        low = kk[None] <= kk[:, None]
        inv = [next(j for j in range(p.nst) if np.allclose(p.sml[P] @ p.sml[j], np.eye(self.n))) for P in range(p.nst)]
        H, S, T, aH, aT = (np.zeros((K, K), LD) for _ in range(5))
        gA, gs, gD = np.zeros((2, K, self.n, self.n), LD), np.zeros((2, K, self.n, 3), LD), np.zeros((2, K), LD)
        for P in range(p.nst):
            m, w = p.sml[P].astype(LD), LD(p.scvv[P])
            Al, sl = self.ket(P)
            ov, tk, er, zh, bra, ket = self.pairs(self.A[:, None], self.s[:, None], self.det[:, None], Al[None], sl[None], self.det[None])
            h = tk + er - zh
            for o, x in ((H, h), (S, ov), (T, tk), (aH, np.abs(tk) + np.abs(er) + np.abs(zh)), (aT, np.abs(tk))):
                o += (w if o is not aH and o is not aT else abs(w)) * x * low
            wb = (2 * w * self.C)[None, :] * low
            wk = (2 * self.C * LD(p.scvv[inv[P]]))[:, None] * (kk[None] < kk[:, None])
            for i, x in enumerate((h, ov)):
                gA[i] += (wb[..., None, None] * bra[i][0]).sum(1) + m @ (wk[..., None, None] * ket[i][0]).sum(0) @ m.T
                gs[i] += (wb[..., None, None] * bra[i][1]).sum(1)
                gs[i] += (p.sms[P].astype(LD).T @ (wk[..., None, None] * ket[i][1]).sum(0).reshape(K, -1).T).T.reshape(K, self.n, 3)
                gD[i] += LD(0.75) * ((wb * x).sum(1) + (wk * x).sum(0))
        full = lambda X: np.tril(X) + np.tril(X, -1).T  # noqa: E731
        H, S, T, aH, aT = (full(X) for X in (H, S, T, aH, aT))
        cSc = self.C @ S @ self.C
        E = (self.C @ H @ self.C) / cSc
        sc = (self.C / cSc)[:, None]
        g = np.concatenate([sc * self.vech(gA[0] - E * gA[1], gD[0] - E * gD[1], self.L), sc * (gs[0] - E * gs[1]).reshape(K, -1)], 1)
        return {"E": E, "g": g, "gC": 2 * (H @ self.C - E * (S @ self.C)) / cSc, "H": H, "S": S, "T": T, "aH": aH, "aT": aT}

    def terms(self, terms):
        """matel and gradel of a list of 1-based (stf, ii, jj): (count, 4), and dh, dov (count, blk)."""
        mat, out = [], ([], [])
        for stf, ii, jj in np.asarray(terms):
            Al, sl = self.ket(stf - 1)
            k, l = ii - 1, jj - 1
            one = lambda x: x[None]  # noqa: E731
            ov, tk, er, zh, bra, _ = self.pairs(*(one(x) for x in (self.A[k], self.s[k], self.det[k], Al[l], sl[l], self.det[l])))
            mat.append([ov[0], tk[0], er[0], zh[0]])
            f = 2 if k == l else 1
            for o, (G, ds), x in zip(out, bra, (tk + er - zh, ov)):
                o.append(f * np.concatenate([self.vech(G, LD(0.75) * x, self.L[k][None])[0], ds.reshape(-1)]))
        return np.array(mat), np.array(out[0]), np.array(out[1])
