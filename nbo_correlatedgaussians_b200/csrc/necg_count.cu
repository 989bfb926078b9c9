// necg_count.cu -- FP64 operation counts of one (k, l, P) term.
//
// Two measures.  `which` 0 .. 3 (energy, ordered gradient, symmetric, fused): the
// direct formulation, in which every term forms its own complete bra and ket
// gradients -- a fixed measure of a term's work, by which rates are quoted and
// compared across versions of the kernels.  `which` 4 .. 7: what the kernels
// execute per term, from the term templates of necg_math.cuh instantiated on the
// host with a counting scalar (every add, subtract and multiply counts 1, so a
// fused multiply-add counts 2; every division, square root, reciprocal,
// reciprocal square root and exponential counts 1 in a separate "special"
// tally; negation and comparisons are free).  They take fewer, because what
// depends on one basis function alone multiplies its sums over all terms.
// Both exclude the per-basis and per-(l, P) work, which is amortised over K terms.
#include <math.h>
#include <stdlib.h>

#include <vector>

#include "necg_math.cuh"
#include "necg_hostscalar.cuh"
#include "../../include/necg.h"

namespace necg {

// Build one bra record (K = 1) and one ket record from a well-conditioned pair.
template <int N> void host_records(std::vector<double> &bra, std::vector<double> &ket) {
    using BL = BraLayout<N>;
    using KL = KetLayout<N>;
    bra.assign(BL::size, 0.0);
    ket.assign(KL::size, 0.0);
    double A[tri(N)], Ap[tri(N)];
    for (int i = 0; i < N; ++i)
        for (int j = 0; j <= i; ++j) {
            A[sx(i, j)] = (i == j) ? 1.0 + 0.1 * i : 0.05;
            Ap[sx(i, j)] = (i == j) ? 0.8 + 0.2 * i : -0.03;
        }
    for (int t = 0; t < tri(N); ++t) {
        bra[BL::A + t] = A[t];
        bra[BL::N8 + t] = -4.0 * A[t];
        bra[BL::L + t] = A[t];
        ket[KL::Ap + t] = Ap[t];
        ket[KL::Np8 + t] = -4.0 * Ap[t];
    }
    for (int t = 0; t < 3 * N; ++t) {
        bra[BL::S + t] = 0.01 * (t + 1);
        bra[BL::AS + t] = 0.02 * (t + 1);
        ket[KL::Sp + t] = -0.01 * (t + 2);
        ket[KL::ASp + t] = -0.015 * (t + 2);
    }
    bra[BL::i1] = 0.01;
    bra[BL::pre] = 1.0;
    bra[BL::tMA] = 2.0;
    ket[KL::i2] = 0.02;
    ket[KL::pre] = 1.0;
    ket[KL::tMA] = 1.0;
    ket[KL::w] = 1.0;
    ket[KL::wC] = 1.0;
    ket[KL::winv] = 1.0;
}

// A term's output as the passes take it: the weighted raw values added to the
// bra's sums and, with KET, scaled for the ket (S too, unless KE).  The ket's
// sum over the warp is counted per (l, P), not per term.
template <int N, bool KET, bool KE> struct CountOut {
    static constexpr bool kets = KET, ket_s = KET && !KE;
    CD acc[2][64], ket[2][64], wb = CD(1.0), wk = CD(1.0), wob, wok;
    NECG_HD void begin(CD ov) {
        wob = wb * ov;
        if (KET) wok = wk * ov;
    }
    NECG_HD void put(int m, int f, CD v) { acc[m][f] += wob * v; }
    NECG_HD void sb1(int f, CD v) { put(1, f, v); }
    NECG_HD void hb1(int f, CD v) { put(0, f, v); }
    template <int I> NECG_HD void sb(CD va, CD vb) {
        put(1, RawPairs<N>::fa(I), va);
        put(1, RawPairs<N>::fb(I), vb);
    }
    template <int I> NECG_HD void hb(CD va, CD vb) {
        put(0, RawPairs<N>::fa(I), va);
        put(0, RawPairs<N>::fb(I), vb);
    }
    template <int I> NECG_HD void sk(CD va, CD vb) {
        ket[1][RawPairs<N>::fa(I)] = wok * va;
        ket[1][RawPairs<N>::fb(I)] = wok * vb;
    }
    template <int I> NECG_HD void hk(CD va, CD vb) {
        ket[0][RawPairs<N>::fa(I)] = wok * va;
        ket[0][RawPairs<N>::fb(I)] = wok * vb;
    }
    NECG_HD void scalar(CD e2) {
        put(0, tri(N), e2);
        acc[1][tri(N)] += wob;
        if (KET) ket[0][tri(N)] = wok * e2;
    }
};

template <int N> void count_term(int which, long long &flops, long long &special) {
    std::vector<double> bra, ket;
    host_records<N>(bra, ket);
    Consts<N> cs;
    for (int i = 0; i < N * N; ++i) cs.M[i] = (i % (N + 1) == 0) ? 0.5 : 0.01;
    for (int t = 0; t < tri(N); ++t) cs.cv[t] = 1.0;
    for (int i = 0; i < N; ++i) cs.q[i] = -1.0;
    cs.efs = 1e-4;
    cs.sqrt8n = ::sqrt(::pow(8.0, N));
    HostBra b{bra.data(), 1};
    HostKet kr{ket.data()};
    count_ctx() = CountCtx();
    if (which == 0) {
        CD ov, t2, rho, sig;
        term_value<N>(b, kr, cs, ov, t2, rho, sig);
        // the energy kernel's per-term accumulation: h and s
        CD w(1.0), h(0.0), s(0.0);
        const CD wov = w * ov;
        h += wov * (t2 + rho - sig);
        s += wov;
    } else if (which == 1) {
        CountOut<N, false, false> out;
        CD eta2, ov;
        term_raw<N>(b, kr, cs, CD(0.0), out, eta2, ov);
    } else if (which == 2) {
        CountOut<N, true, true> out;
        CD eta2, ov;
        term_raw<N>(b, kr, cs, CD(0.5), out, eta2, ov);
    } else {
        CountOut<N, true, false> out;
        CD eta2, ov, hs(0.0), ss(0.0), w(1.0);
        term_raw<N>(b, kr, cs, CD(0.0), out, eta2, ov);
        const CD wo = w * ov;  // the pass's sums of w_P h and w_P ov over P
        hs += wo * eta2;
        ss += wo;
    }
    flops = count_ctx().flops;
    special = count_ctx().special;
}

}  // namespace necg

namespace {
// direct formulation: total operations (special ones included) by n and which;
// the special ones are two per Coulomb pair, one per Cholesky pivot and the exponential
const int kDirect[6][4] = {{93, 201, 253, 281},      {249, 585, 743, 795},     {496, 1206, 1547, 1626},
                           {819, 2067, 2686, 2795}, {1254, 3222, 4232, 4374}, {1795, 4683, 6215, 6393}};
}  // namespace

extern "C" long long necg_term_flops(int n, int which, long long *special) {
    long long f = 0, s = 0;
    if (n < 1 || n > 6 || which < 0 || which > 7) return -1;
    if (which < 4) {
        if (special) *special = n * (n + 1) + n + 1;
        return kDirect[n - 1][which];
    }
    switch (n) {
    case 1: necg::count_term<1>(which - 4, f, s); break;
    case 2: necg::count_term<2>(which - 4, f, s); break;
    case 3: necg::count_term<3>(which - 4, f, s); break;
    case 4: necg::count_term<4>(which - 4, f, s); break;
    case 5: necg::count_term<5>(which - 4, f, s); break;
    default: necg::count_term<6>(which - 4, f, s); break;
    }
    if (special) *special = s;
    return f + s;
}
