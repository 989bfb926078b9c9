// necg_emu.cu -- TEST INFRASTRUCTURE: runs the per-thread bodies
// (nbo_correlatedgaussians_b200/csrc/necg_lanes.cuh) of the kernels whose lanes work
// alone (energy and ordered gradient tiles, single terms, the dipole) on the host,
// lane by lane and tile by tile, so the CPU test suite can check the device algorithm
// against the oracle without a GPU.  The passes over unordered pairs, whose warps
// work together, are run by simt_emu.cpp.  Never linked into the product library.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "../../nbo_correlatedgaussians_b200/csrc/necg_hostscalar.cuh"
#include "../../nbo_correlatedgaussians_b200/csrc/necg_lanes.cuh"
#include "../../nbo_correlatedgaussians_b200/csrc/necg_tiles.h"

using namespace necg;

namespace {

template <int N> Consts<N> consts(const double *mass, const double *ncv, double efs) {
    Consts<N> c;
    for (int i = 0; i < N * N; ++i) c.M[i] = mass[i];
    for (int q = 1; q <= N; ++q)
        for (int p = 0; p < q; ++p) c.cv[vidx(p, q)] = 2.0 * ncv[p] * ncv[q] / NECG_SQRT_PI;
    for (int i = 0; i < N; ++i) c.q[i] = ncv[i + 1];
    c.efs = efs;
    c.sqrt8n = ::sqrt(::pow(8.0, N));
    return c;
}

// Accumulators of one bra gradient (SmemAcc on the device).
template <int N> struct RegAcc {
    CD G[tri(N)], D, S[3 * N];
    NECG_HD void zero() {
        for (CD &v : G) v = CD(0.0);
        D = CD(0.0);
        for (CD &v : S) v = CD(0.0);
    }
    NECG_HD CD &g(int t) { return G[t]; }
    NECG_HD CD &d() { return D; }
    NECG_HD CD &s(int t) { return S[t]; }
};

struct Args {
    int nst, K;
    double efs;
    const double *mass, *ncv, *scvv, *sml, *sms;
};

template <int N>
void prep(const Args &a, const double *iv, const double *C, std::vector<double> &bra,
          std::vector<double> &ket, const Consts<N> &cs) {
    bra.assign((size_t)BraLayout<N>::size * a.K, 0.0);
    ket.assign((size_t)KetLayout<N>::size * a.K * a.nst, 0.0);
    for (int k = 0; k < a.K; ++k) prep_bra_at<N>(iv + (size_t)k * (tri(N) + 3 * N), cs, bra.data() + k, (size_t)a.K);
    for (int id = 0; id < a.K * a.nst; ++id)
        prep_ket_one<N>(iv, C, a.nst, cs, a.sml, a.sms, a.scvv, ket.data(), id);
}

template <int N>
int outprod(const Args &a, const double *x, int LCe, int LCg, double *f, double *g, double *H,
            double *S) {
    const int K = a.K, nst = a.nst;
    const size_t siv = (size_t)K * (tri(N) + 3 * N);
    const double *iv = x, *C = x + siv;
    Consts<N> cs = consts<N>(a.mass, a.ncv, a.efs);
    std::vector<double> bra, ket;
    prep<N>(a, iv, C, bra, ket, cs);
    int flags = 0;
    // energy tiles in the order of the device tile list
    for (int kb = 0; kb * 32 < K; ++kb)
        for (int lc = 0; lc * LCe <= kb * 32 + 31 && lc * LCe < K; ++lc)
            for (int lane = 0; lane < 32; ++lane) {
                int k, l0, lend, bad = 0;
                if (!energy_lane_range(kb, lc, lane, LCe, K, k, l0, lend)) continue;
                flags |= energy_lane<N, CD>(HostBra{bra.data() + k, (size_t)K},
                                            HostKetBase{ket.data()}, k, l0, lend, K, nst, cs, H, S,
                                            nullptr, nullptr, bad);
            }
    // rows + finalize
    std::vector<double> rh(K), rs(K);
    for (int i = 0; i < K; ++i) {
        double h = 0.0, s = 0.0;
        for (int j = 0; j < K; ++j) {
            h += H[(size_t)i * K + j] * C[j];
            s += S[(size_t)i * K + j] * C[j];
        }
        rh[i] = h;
        rs[i] = s;
    }
    double cHc = 0.0, cSc = 0.0;
    for (int i = 0; i < K; ++i) {
        cHc += C[i] * rh[i];
        cSc += C[i] * rs[i];
    }
    const double E = cHc / cSc, norm = 1.0 / cSc;
    *f = E;
    for (int i = 0; i < K; ++i) g[siv + i] = 2.0 * norm * (rh[i] - E * rs[i]);
    // gradient tiles
    const int nkb = (K + 31) / 32, nlc = (K + LCg - 1) / LCg;
    std::vector<double> part((size_t)Part<N>::size * K * nlc, 0.0);
    for (int w = 0; w < nkb * nlc; ++w)
        for (int lane = 0; lane < 32; ++lane) {
            int k, lc, l0, l1;
            if (!grad_lane_range(w, lane, nkb, LCg, K, k, lc, l0, l1)) continue;
            RegAcc<N> accH, accS;
            if (!grad_lane<N, CD>(HostBra{bra.data() + k, (size_t)K}, HostKetBase{ket.data()}, l0, l1,
                                  nst, cs, CD(1.0), CD(E), part.data() + (size_t)lc * Part<N>::size * K + k,
                                  (size_t)K, accH, accS))
                flags |= 1;
        }
    for (int k = 0; k < K; ++k)
        if (!grad_reduce_at<N>(part.data(), nlc, K, bra.data() + k, (size_t)K, norm * C[k], g, k)) flags |= 2;
    return flags;
}

// Host mirror of rrms_kernel (per term) and of dipole_kernel + dipole_sum_kernel
// (energy tiles in the device list order, per-lane sums over (Pe, l, P), the
// warp's butterfly sum, tile partials summed by 256 strided threads and a tree).
template <int N> int rrms_terms(const Args &a, const double *iv, int nterms, const int *terms, double *out) {
    using KL = KetLayout<N>;
    Consts<N> cs = consts<N>(a.mass, a.ncv, a.efs);
    std::vector<double> bra, ket;
    prep<N>(a, iv, nullptr, bra, ket, cs);
    int flags = 0;
    for (int t = 0; t < nterms; ++t) {
        const int *q = terms + 5 * t;
        const int stfe = q[0] - 1, stf = q[1] - 1, ii = q[2] - 1, jj = q[3] - 1, n1 = q[4] - 1;
        CD T[3 * N], ov;
        if (!term_dipole<N, CD>(HostKet{ket.data() + ((size_t)ii * a.nst + stfe) * KL::size},
                                HostKet{ket.data() + ((size_t)jj * a.nst + stf) * KL::size}, cs, T, ov))
            flags |= 1;
        out[2 * t] = ov.v;
        out[2 * t + 1] = T[n1].v * ov.v;
    }
    return flags;
}

template <int N> int dipole(const Args &a, const double *iv, const double *C, int LC, double *comps, double *dip) {
    using KL = KetLayout<N>;
    constexpr int NM = 3 * N + 1;
    const int K = a.K, nst = a.nst;
    Consts<N> cs = consts<N>(a.mass, a.ncv, a.efs);
    std::vector<double> bra, ket;
    prep<N>(a, iv, C, bra, ket, cs);
    int flags = 0;
    std::vector<double> part;
    for (int kb = 0; kb * 32 < K; ++kb)
        for (int lc = 0; lc * LC <= kb * 32 + 31 && lc * LC < K; ++lc) {
            double acc[32][NM] = {};
            for (int lane = 0; lane < 32; ++lane) {
                int k, l0, lend;
                if (!energy_lane_range(kb, lc, lane, LC, K, k, l0, lend)) continue;
                for (int Pe = 0; Pe < nst; ++Pe) {
                    const double *kbr = ket.data() + ((size_t)k * nst + Pe) * KL::size;
                    const double wek = kbr[KL::w] * C[k];
                    for (int l = l0; l < lend; ++l) {
                        const double wl = (l == k ? 1.0 : 2.0) * wek * C[l];
                        for (int P = 0; P < nst; ++P) {
                            const double *kr = ket.data() + ((size_t)l * nst + P) * KL::size;
                            CD T[3 * N], ov;
                            if (!term_dipole<N, CD>(HostKet{kbr}, HostKet{kr}, cs, T, ov)) flags |= 1;
                            const double wo = wl * kr[KL::w] * ov.v;
                            acc[lane][0] += wo;
                            for (int m = 0; m < 3 * N; ++m) acc[lane][1 + m] += wo * T[m].v;
                        }
                    }
                }
            }
            for (int m = 0; m < NM; ++m) {  // butterfly: xor 16, 8, 4, 2, 1
                double v[32];
                for (int lane = 0; lane < 32; ++lane) v[lane] = acc[lane][m];
                for (int o = 16; o > 0; o >>= 1) {
                    double w[32];
                    for (int lane = 0; lane < 32; ++lane) w[lane] = v[lane] + v[lane ^ o];
                    for (int lane = 0; lane < 32; ++lane) v[lane] = w[lane];
                }
                part.push_back(v[0]);
            }
        }
    const int ntiles = (int)(part.size() / NM);
    double tot[NM];
    for (int m = 0; m < NM; ++m) {
        double red[256];
        for (int j = 0; j < 256; ++j) {
            double s = 0.0;
            for (int t = j; t < ntiles; t += 256) s += part[(size_t)t * NM + m];
            red[j] = s;
        }
        for (int w = 128; w > 0; w >>= 1)
            for (int j = 0; j < w; ++j) red[j] += red[j + w];
        tot[m] = red[0];
    }
    for (int m = 0; m < 3 * N; ++m) comps[m] = tot[0] != 0.0 ? tot[1 + m] / tot[0] : 0.0;
    for (int c = 0; c < 3; ++c) {
        double d = 0.0;
        for (int i = 0; i < N; ++i) d += cs.q[i] * comps[3 * i + c];
        dip[c] = d;
    }
    return flags;
}

template <int N>
int elements(const Args &a, const double *iv, int nterms, const int *terms, double *mat,
             double *tg, double *tgs) {
    constexpr int blk = tri(N) + 3 * N;
    Consts<N> cs = consts<N>(a.mass, a.ncv, a.efs);
    std::vector<double> bra, ket;
    prep<N>(a, iv, nullptr, bra, ket, cs);
    int flags = 0;
    for (int t = 0; t < nterms; ++t) {
        const int stf = terms[3 * t] - 1, ii = terms[3 * t + 1] - 1, jj = terms[3 * t + 2] - 1;
        const HostKet kr{ket.data() + ((size_t)jj * a.nst + stf) * KetLayout<N>::size};
        const HostBra b{bra.data() + ii, (size_t)a.K};
        if (!matel_one<N, CD>(b, kr, cs, mat + 4 * t)) flags |= 1;
        double L[tri(N)];
        for (int q = 0; q < tri(N); ++q) L[q] = bra[(BraLayout<N>::L + q) * (size_t)a.K + ii];
        if (!gradel_one<N, CD>(b, kr, cs, L, ii == jj, tg + (size_t)t * blk, tgs + (size_t)t * blk))
            flags |= 1;
    }
    return flags;
}

}  // namespace

#define EMU_DISPATCH(n, expr)               \
    switch (n) {                            \
    case 1: { constexpr int N = 1; return expr; } \
    case 2: { constexpr int N = 2; return expr; } \
    case 3: { constexpr int N = 3; return expr; } \
    case 4: { constexpr int N = 4; return expr; } \
    case 5: { constexpr int N = 5; return expr; } \
    case 6: { constexpr int N = 6; return expr; } \
    default: return -1;                     \
    }

extern "C" int emu_outprod(int n, int nst, int K, double efs, const double *mass, const double *ncv,
                           const double *scvv, const double *sml, const double *sms, const double *x,
                           int lc_e, int lc_g, double *f, double *g, double *H, double *S) {
    Args a{nst, K, efs, mass, ncv, scvv, sml, sms};
    EMU_DISPATCH(n, (outprod<N>(a, x, lc_e, lc_g, f, g, H, S)));
}

extern "C" int emu_rrms(int n, int nst, int K, double efs, const double *mass, const double *ncv,
                        const double *scvv, const double *sml, const double *sms, const double *iv, int nterms,
                        const int *terms, double *out) {
    Args a{nst, K, efs, mass, ncv, scvv, sml, sms};
    EMU_DISPATCH(n, (rrms_terms<N>(a, iv, nterms, terms, out)));
}

extern "C" int emu_dipole(int n, int nst, int K, double efs, const double *mass, const double *ncv,
                          const double *scvv, const double *sml, const double *sms, const double *iv,
                          const double *C, int lc, double *comps, double *dip) {
    Args a{nst, K, efs, mass, ncv, scvv, sml, sms};
    EMU_DISPATCH(n, (dipole<N>(a, iv, C, lc, comps, dip)));
}

extern "C" int emu_elements(int n, int nst, int K, double efs, const double *mass, const double *ncv,
                            const double *scvv, const double *sml, const double *sms, const double *iv,
                            int nterms, const int *terms, double *mat, double *tg, double *tgs) {
    Args a{nst, K, efs, mass, ncv, scvv, sml, sms};
    EMU_DISPATCH(n, (elements<N>(a, iv, nterms, terms, mat, tg, tgs)));
}

// A M A (packed lower) and tr(M A) of every function as the bra's and as the kets'
// records hold them: bra K x (tri + 1), ket K x nst x (tri + 1).
namespace {
template <int N> int mass_records(const Args &a, const double *iv, double *ob, double *ok) {
    std::vector<double> bra, ket;
    Consts<N> cs = consts<N>(a.mass, a.ncv, a.efs);
    prep<N>(a, iv, nullptr, bra, ket, cs);
    for (int k = 0; k < a.K; ++k)
        for (int t = 0; t <= tri(N); ++t) {
            ob[k * (tri(N) + 1) + t] = bra[(size_t)(t < tri(N) ? BraLayout<N>::N8 + t : BraLayout<N>::tMA) * a.K + k];
            for (int P = 0; P < a.nst; ++P)
                ok[((size_t)k * a.nst + P) * (tri(N) + 1) + t] =
                    ket[((size_t)k * a.nst + P) * KetLayout<N>::size + (t < tri(N) ? KetLayout<N>::Np8 + t : KetLayout<N>::tMA)];
        }
    return 0;
}
}  // namespace
extern "C" int emu_mass_records(int n, int nst, int K, double efs, const double *mass, const double *ncv,
                                const double *scvv, const double *sml, const double *sms, const double *iv, double *ob,
                                double *ok) {
    Args a{nst, K, efs, mass, ncv, scvv, sml, sms};
    EMU_DISPATCH(n, (mass_records<N>(a, iv, ob, ok)));
}

// The tile lists of the symmetric passes, filled row block by row block with nj
// threads each; head: ntiles, units, groups of 8, tail0, ntail, parts.  Null lists: head only.
extern "C" int emu_sym_lists(int K, int LC, int w, int nst, int sms, int nj, int *head, int *tiles, int *start,
                             int *groups, int *urange, int *tslot, int *bgroups, int *burange) {
    const SymQueue q = sym_queue(K, LC, w, nst, sms);
    const int h[6] = {q.ntiles, q.units(), groups_before(K, LC, 8, -1), q.tail0, q.ntail, q.parts};
    for (int i = 0; i < 6; ++i) head[i] = h[i];
    if (!tiles) return 0;
    const SymLists o{(int2 *)tiles, start, (int2 *)groups, (int2 *)urange, tslot, (int2 *)bgroups, (int2 *)burange};
    for (int kb = 0; kb < row_blocks(K); ++kb)
        for (int j = 0; j < nj; ++j) fill_sym_lists(q, o, kb, j, nj);
    return 0;
}
