// necg_lanes.cuh -- per-thread bodies of the kernels, shared by the CUDA
// kernels (R = double, device accessors) and by the host-side test emulator
// (R = a value-carrying scalar, host accessors), so that the emulator exercises
// exactly the index arithmetic, loop bounds and reductions the kernels run.
#pragma once
#include "necg_math.cuh"

namespace necg {

NECG_HD double val(double x) { return x; }

// Unpack vech(L) (python/matel.py:59-66: column-major lower triangle) into a
// packed-lower row-major array.
template <int N> NECG_HD void unpack_L(const double *blk, double (&L)[tri(N)]) {
    int idx = 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = j; i < N; ++i) L[sx(i, j)] = blk[idx++];
}

// A = L L^T (packed)
template <int N> NECG_HD void llt(const double (&L)[tri(N)], double (&A)[tri(N)]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k <= j; ++k) s += L[sx(i, k)] * L[sx(j, k)];
            A[sx(i, j)] = s;
        }
}

// A M (full), A M A (packed) and tr(M A)
template <int N>
NECG_HD void mass_products(const double (&A)[tri(N)], const double *M, double (&AM)[N * N],
                           double (&AMA)[tri(N)], double &tMA) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += A[sx(i, k)] * M[k * N + j];
            AM[i * N + j] = s;
        }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += AM[i * N + k] * A[sx(k, j)];
            AMA[sx(i, j)] = s;
        }
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) t += AM[i * N + i];
    tMA = t;
}

// Bra record of the basis function with parameters b: field f at bra[f * stride].
template <int N>
NECG_HD void prep_bra_at(const double *b, const Consts<N> &cs, double *bra, size_t stride) {
    using BL = BraLayout<N>;
    double L[tri(N)], A[tri(N)], S[3 * N], AS[3 * N], AM[N * N], AMA[tri(N)], tMA;
    unpack_L<N>(b, L);
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) S[t] = b[tri(N) + t];
    llt<N>(L, A);
    symv3<N>(A, 0, S, AS);
    mass_products<N>(A, cs.M, AM, AMA, tMA);
    double i1 = 0.0, dl = 1.0;
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) i1 += S[t] * AS[t];
#pragma unroll
    for (int i = 0; i < N; ++i) dl *= L[sx(i, i)];
    dl = ::fabs(dl);
#pragma unroll
    for (int t = 0; t < tri(N); ++t) bra[(BL::A + t) * stride] = A[t];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) bra[(BL::S + t) * stride] = S[t];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) bra[(BL::AS + t) * stride] = AS[t];
#pragma unroll
    for (int t = 0; t < tri(N); ++t) bra[(BL::N8 + t) * stride] = -8.0 * AMA[t];
    bra[BL::i1 * stride] = i1;
    bra[BL::pre * stride] = cs.sqrt8n * (dl * ::sqrt(dl));
    bra[BL::tMA * stride] = tMA;
#pragma unroll
    for (int t = 0; t < tri(N); ++t) bra[(BL::L + t) * stride] = L[t];
}

// Ket record of (l, P) = id / nst, id % nst: python/matel.py:76-87
// (al <- sml^T al sml, st2 <- sms st2) plus the data the tiles reuse.  general =
// false: the shift map is kron(m, I3), so that m alone is read (25 instead of 225
// entries at n = 5).
template <int N>
NECG_HD void prep_ket_one(const double *iv, const double *C, int nst, const Consts<N> &cs,
                          const double *sml, const double *sms, const double *scvv, double *ket,
                          int id, const int *pinv = nullptr, bool general = true) {
    using KL = KetLayout<N>;
    constexpr int blk = tri(N) + 3 * N;
    const int l = id / nst, P = id - l * nst;
    const double *b = iv + (size_t)l * blk;
    double L[tri(N)], A[tri(N)];
    unpack_L<N>(b, L);
    llt<N>(L, A);
    const double *pm = sml + (size_t)P * N * N;
    double Apm[N * N];  // A pm
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += A[sx(i, k)] * pm[k * N + j];
            Apm[i * N + j] = s;
        }
    double Ap[tri(N)];  // pm^T A pm
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += pm[k * N + i] * Apm[k * N + j];
            Ap[sx(i, j)] = s;
        }
    const double *sm = sms + (size_t)P * 9 * N * N;  // 3n x 3n shift map
    double Sp[3 * N];
    if (general) {
#pragma unroll
        for (int r = 0; r < 3 * N; ++r) {
            double s = 0.0;
#pragma unroll
            for (int c = 0; c < 3 * N; ++c) s += sm[r * 3 * N + c] * b[tri(N) + c];
            Sp[r] = s;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const double m = sm[(3 * i) * 3 * N + 3 * j];
#pragma unroll
                for (int c = 0; c < 3; ++c) s[c] += m * b[tri(N) + 3 * j + c];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) Sp[3 * i + c] = s[c];
        }
    }
    double ASp[3 * N];
    symv3<N>(Ap, 0, Sp, ASp);
    double i2 = 0.0, dl = 1.0;
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) i2 += Sp[t] * ASp[t];
#pragma unroll
    for (int i = 0; i < N; ++i) dl *= L[sx(i, i)];
    dl = ::fabs(dl);
    double *o = ket + (size_t)id * KL::size;
#pragma unroll
    for (int t = 0; t < tri(N); ++t) o[KL::Ap + t] = Ap[t];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) o[KL::ASp + t] = ASp[t];
    o[KL::i2] = i2;
    o[KL::pre] = dl * ::sqrt(dl);
    o[KL::w] = scvv[P];
    o[KL::wC] = C ? 2.0 * scvv[P] * C[l] : 0.0;
    o[KL::winv] = pinv ? scvv[pinv[P]] : 0.0;
    // A' M A' = pm^T (A (pm M pm^T) A) pm, and the trace likewise: where M is
    // unchanged by pm, as in a permutation of equal particles, these are the bra's own
    // values in another order, with the same rounding for every P, which then
    // cancels in an antisymmetric sum over P as the terms do (E of LiH K = 512: 1e-14
    // relative with A' M A' formed from A', 1e-15 so)
    double Mp[N * N], AM[N * N], AMA[tri(N)], tMA;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double r[N];  // row i of pm M
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += pm[i * N + k] * cs.M[k * N + j];
            r[j] = s;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += r[k] * pm[j * N + k];
            Mp[i * N + j] = s;
        }
    }
    mass_products<N>(A, Mp, AM, AMA, tMA);
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += AMA[sx(i, k)] * pm[k * N + j];
            AM[i * N + j] = s;  // A Mp A pm
        }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k) s += pm[k * N + i] * AM[k * N + j];
            o[KL::Np8 + sx(i, j)] = -8.0 * s;
        }
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) o[KL::Sp + t] = Sp[t];
    o[KL::tMA] = tMA;
    if (KL::size > KL::Sp + 3 * N) o[KL::Sp + 3 * N] = 0.0;
}

// Sums over the symmetry terms [p0, p1) of one pair: sum[0] = H, [1] = S, [2] =
// kinetic, [3] = Coulomb; false if some B is not positive definite.
template <int N, typename R, typename BA, typename KB>
NECG_HD bool energy_sums(const BA &b, const KB &ket, int l, int nst, int p0, int p1, const Consts<N> &cs,
                         R (&sum)[4]) {
    using KL = KetLayout<N>;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] = R(0.0);
    for (int P = p0; P < p1; ++P) {
        const auto kr = ket.at(((size_t)l * nst + P) * KL::size);
        R ov, t2, rho, sig;
        ok = term_value<N>(b, kr, cs, ov, t2, rho, sig) && ok;
        const R wov = kr[KL::w] * ov;
        sum[0] += wov * (t2 + rho - sig);
        sum[1] += wov;
        sum[2] += wov * t2;
        sum[3] += wov * rho;
    }
    return ok;
}

// Write one pair's sums to H, S (and Kin, Pot when non-null) symmetrically; returns
// the status flags (1: not positive definite, 2: non-finite).
NECG_HD int energy_store(const double (&v)[4], bool ok, int k, int l, int K, double *H, double *S, double *Kin,
                         double *Pot) {
    double *M[4] = {H, S, Kin, Pot};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (M[i]) {
            M[i][(size_t)k * K + l] = v[i];
            M[i][(size_t)l * K + k] = v[i];
        }
    return (ok ? 0 : 1) | (isfinite(v[0]) && isfinite(v[1]) ? 0 : 2);
}

// Energy tile lane: bra k against kets l in [l0, lend) (lend <= k + 1), all P.
// Writes H, S (and Kin, Pot when non-null) symmetrically.  Returns status
// flags (1: a pair not positive definite, 2: non-finite) and the first pair.
template <int N, typename R, typename BA, typename KB>
NECG_HD int energy_lane(const BA &b, const KB &ket, int k, int l0, int lend, int K, int nst,
                        const Consts<N> &cs, double *H, double *S, double *Kin, double *Pot,
                        int &bad_pair) {
    int flags = 0;
    for (int l = l0; l < lend; ++l) {
        R sum[4];
        const bool ok = energy_sums<N, R>(b, ket, l, nst, 0, nst, cs, sum);
        const double v[4] = {val(sum[0]), val(sum[1]), val(sum[2]), val(sum[3])};
        const int fl = energy_store(v, ok, k, l, K, H, S, Kin, Pot);
        if (fl && !flags) bad_pair = k * K + l;
        flags |= fl;
    }
    return flags;
}

// Partial-buffer stride (doubles per basis function): dF/dA_k packed, the
// coefficient of A_k^-1 in dF/dA_k, dF/ds_k.
template <int N> struct Part {
    static constexpr int G = 0;
    static constexpr int D = tri(N);
    static constexpr int S = D + 1;
    static constexpr int size = S + 3 * N;
};

// Raw sums of one bra over its terms (term_raw's `out`): H and S fields into two
// accumulators (g(t), d(), s(t)), weight w ov.
template <int N, typename R, typename ACC> struct BraSums {
    static constexpr bool kets = false, ket_s = false;
    ACC &H, &S;
    R w, wo;
    NECG_HD static R &at(ACC &a, int f) { return f < tri(N) ? a.g(f) : f == tri(N) ? a.d() : a.s(f - tri(N) - 1); }
    NECG_HD void begin(R ov) { wo = w * ov; }
    NECG_HD void sb1(int f, R v) { at(S, f) += wo * v; }
    NECG_HD void hb1(int f, R v) { at(H, f) += wo * v; }
    template <int I> NECG_HD void sb(R va, R vb) {
        sb1(RawPairs<N>::fa(I), va);
        sb1(RawPairs<N>::fb(I), vb);
    }
    template <int I> NECG_HD void hb(R va, R vb) {
        hb1(RawPairs<N>::fa(I), va);
        hb1(RawPairs<N>::fb(I), vb);
    }
    NECG_HD void scalar(R e2) {
        H.d() += wo * e2;
        S.d() += wo;
    }
};

// Gradient tile lane: bra k against kets l in [l0, l1), all P, weights
// wC(l, P) = 2 scvv[P] C_l: the raw sums in accH and accS, then the gradient of
// lam H - E S folded from them into part[f * stride] (f < Part::size).
template <int N, typename R, typename BA, typename KB, typename ACC>
NECG_HD bool grad_lane(const BA &b, const KB &ket, int l0, int l1, int nst, const Consts<N> &cs,
                       R lam, R E, double *part, size_t stride, ACC &accH, ACC &accS) {
    using KL = KetLayout<N>;
    using BL = BraLayout<N>;
    constexpr int PS = Part<N>::size;
    accH.zero();
    accS.zero();
    bool ok = true;
    BraSums<N, R, ACC> sums{accH, accS, R(0.0), R(0.0)};
    for (int l = l0; l < l1; ++l)
        for (int P = 0; P < nst; ++P) {
            const auto kr = ket.at(((size_t)l * nst + P) * KL::size);
            sums.w = R(kr[KL::wC]);
            R eta2, ov;
            ok = term_raw<N>(b, kr, cs, R(0.0), sums, eta2, ov) && ok;
        }
    R r[PS], o[PS];
    const auto sr = [&](int f) { return BraSums<N, R, ACC>::at(accS, f); };
    const auto A = [&](int t) { return b(BL::A + t); };
#pragma unroll
    for (int f = 0; f < PS; ++f) r[f] = BraSums<N, R, ACC>::at(accH, f);
    explicit_tau<N>(sr, A, cs, r);
#pragma unroll
    for (int f = 0; f < PS; ++f) r[f] = lam * r[f] - 2.0 * E * sr(f);
    fold_raw<N>(FieldsOf<R>{r}, A, o);
#pragma unroll
    for (int f = 0; f < PS; ++f) part[f * stride] = val(o[f]);
    return ok;
}

// Map an A-space gradient dF/dA = G + D A^-1 (G packed symmetric, D the
// scalar coefficient of A^-1) and dF/ds = gS to the reference's parameter
// block [vech(dF/dL), dF/ds]: dF/dL = 2 (G + D A^-1) L = 2 G L + 2 D L^-T, whose
// lower triangle is 2 (G L)_ij for i > j and 2 (G L)_ii + 2 D / L_ii on the
// diagonal.  out[blk] scaled by sc.
template <int N>
NECG_HD bool a_to_vech(const double (&G)[tri(N)], double D, const double (&gS)[3 * N],
                       const double (&L)[tri(N)], double sc, double *out) {
    int idx = 0;
    bool fin = true;
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = j; i < N; ++i) {
            double s = 0.0;  // (G L)_ij = sum_{a >= j} G_ia L_aj
#pragma unroll
            for (int a = j; a < N; ++a) s += G[sx(i, a)] * L[sx(a, j)];
            s *= 2.0;
            if (i == j) s += 2.0 * D / L[sx(i, i)];
            const double v = sc * s;
            fin = fin && isfinite(v);
            out[idx++] = v;
        }
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) {
        const double v = sc * gS[t];
        fin = fin && isfinite(v);
        out[tri(N) + t] = v;
    }
    return fin;
}

// Sum the nlc partials of basis k and write its GRADA block scaled by sc; brak:
// field f of its bra record at brak[f * stride].
template <int N>
NECG_HD bool grad_reduce_at(const double *part, int nlc, int K, const double *brak, size_t stride, double sc, double *g,
                            int k) {
    constexpr int PS = Part<N>::size;
    double o[PS];
#pragma unroll
    for (int f = 0; f < PS; ++f) o[f] = 0.0;
    for (int lc = 0; lc < nlc; ++lc) {
        const double *p = part + (size_t)lc * PS * K + k;
#pragma unroll
        for (int f = 0; f < PS; ++f) o[f] += p[(size_t)f * K];
    }
    double G[tri(N)], gS[3 * N], L[tri(N)];
#pragma unroll
    for (int t = 0; t < tri(N); ++t) G[t] = o[t];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) gS[t] = o[tri(N) + 1 + t];
#pragma unroll
    for (int t = 0; t < tri(N); ++t) L[t] = brak[(BraLayout<N>::L + t) * stride];
    return a_to_vech<N>(G, o[tri(N)], gS, L, sc, g + (size_t)k * (tri(N) + 3 * N));
}
// One matel term (python/matel.py:28-210): out = (ov, tk, ert, zht).
template <int N, typename R, typename BA, typename KR>
NECG_HD bool matel_one(const BA &b, const KR &kr, const Consts<N> &cs, double *out) {
    R ov, tau2, rho, sig;
    const bool ok = term_value<N>(b, kr, cs, ov, tau2, rho, sig);
    out[0] = val(ov);
    out[1] = val(ov * tau2);
    out[2] = val(ov * rho);
    out[3] = val(ov * sig);
    return ok;
}

// One gradel term (python/gradel.py:27-392): dH and dS with respect to the bra
// block, doubled when ii == jj (python/gradel.py:388-390).
template <int N, typename R, typename BA, typename KR>
NECG_HD bool gradel_one(const BA &b, const KR &kr, const Consts<N> &cs, const double (&L)[tri(N)],
                        bool diag, double *tgvl, double *tgvls) {
    constexpr int PS = Part<N>::size;
    R bH[PS], bS[PS];
    const bool ok = term_grad<N>(b, kr, cs, bH, bS);
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        const R(&v)[PS] = which == 0 ? bH : bS;
        double G[tri(N)], gS[3 * N];
#pragma unroll
        for (int q = 0; q < tri(N); ++q) G[q] = val(v[q]);
#pragma unroll
        for (int q = 0; q < 3 * N; ++q) gS[q] = val(v[tri(N) + 1 + q]);
        a_to_vech<N>(G, val(v[tri(N)]), gS, L, diag ? 2.0 : 1.0, which == 0 ? tgvl : tgvls);
    }
    return ok;
}

// Energy tiles over the lower triangle: tile (kb, lc) covers the bras of row block
// kb and kets l in [lc LC, lc LC + LC) with l <= k; it has pairs when lc LC <=
// row_last(K, kb).  The count here is of all with lc LC <= 32 kb + 31 and lc LC < K,
// an upper bound, for lists made without looking at K's remainder.
NECG_HD int energy_tile_count(int K, int LC) {
    int n = 0;
    for (int kb = 0; kb * 32 < K; ++kb) {
        const int kmax = kb * 32 + 31;
        const int last = kmax < K - 1 ? kmax : K - 1;
        n += last / LC + 1;
    }
    return n;
}

// Where the pair passes keep the ket's raw fields of a term: field f of matrix
// `which` (0: H or the combined gradient, 1: S) in slot which * SL + slot(f) of a
// table row.  The two fields of a pair (RawPairs) are 8 slots apart, so that the
// even and the odd lanes of a warp, which store one side each, use different
// shared-memory banks (rows are an odd number of doubles apart).
template <int N> struct KetSlots {
    static constexpr int SL = 16 * ((RawPairs<N>::count + 7) / 8);  // slots per matrix (16 or 32 for n <= 5)
    __host__ __device__ static constexpr int of_pair(int i) { return 16 * (i >> 3) + (i & 7); }
    __host__ __device__ static constexpr int slot(int f) {
        return of_pair(RawPairs<N>::pair_of(f)) + 8 * RawPairs<N>::side_of(f);
    }
};

// Sparse linear map of the ket's raw sums from P's transformed frame to the basis
// function's own, by slot: entry (P, slot): cnt values at src/coef[(P * SL + slot)
// * maxnz + i], src a slot of the same matrix.  fold: the set's shift maps are
// not those of its coordinate maps (sms = kron(sml^-1, I3)), so that e' = A' s'
// does not map as e does: the sums are folded into gradients in P's frame
// (fold_raw) and those are mapped, with dF/ds' by sms^T.
struct RawMap {
    const int *cnt, *src;
    const double *coef;
    int maxnz, fold;
};

// Fields the symmetric passes sum per basis function and matrix: the raw fields
// and, last, its row of H C or S C.
template <int N> struct SumFields {
    static constexpr int row = Part<N>::size;
    static constexpr int size = row + 1;
};

// Per-basis sums of the symmetric passes: kSumSets sets of SumFields, field f of
// set i of basis k at (i SumFields::size + f) K + k: the bra's H (or, with E
// known, combined) and S sums, then the ket's.
constexpr int kSumSets = 4;

// Lane ranges of the two tile kinds (used by the kernels and the emulator).
// Energy: tile (kb, lc) -> lane's bra k of row block kb, kets [l0, lend); false if idle.
NECG_HD bool energy_lane_range(int kb, int lc, int lane, int LC, int K, int &k, int &l0, int &lend) {
    k = kb * 32 + lane - row_pad(K);
    l0 = lc * LC;
    if (k < 0 || k >= K || l0 > k) return false;
    lend = l0 + LC < K ? l0 + LC : K;
    if (lend > k + 1) lend = k + 1;
    return true;
}
// Gradient: warp w -> (kb = w % nkb, lc = w / nkb), bra k = 32 kb + lane,
// kets [l0, l1); false if idle.
NECG_HD bool grad_lane_range(int w, int lane, int nkb, int LC, int K, int &k, int &lc, int &l0,
                             int &l1) {
    const int kb = w % nkb;
    lc = w / nkb;
    k = kb * 32 + lane;
    if (k >= K) return false;
    l0 = lc * LC;
    l1 = l0 + LC < K ? l0 + LC : K;
    return true;
}

}  // namespace necg
