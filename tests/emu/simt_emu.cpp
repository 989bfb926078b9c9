// simt_emu.cpp -- TEST INFRASTRUCTURE: the device code of the passes over unordered
// pairs (nbo_correlatedgaussians_b200/csrc/necg_device.cuh) compiled for the host and run
// thread by thread (simt.h): the tiles with their ket tables, slots and maps, the block
// variants with their queue and split tail, the sums and the finish.  What is repeated
// here is only what the kernels' shells do (which block takes what).  Workspaces start
// as NaN, so that a value that nobody wrote shows in the results.
// Built by g++ with tests/emu/stub first in the include path; never linked into the
// product library.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <limits>
#include <vector>

#include "simt.h"

#include "../../nbo_correlatedgaussians_b200/csrc/necg_device.cuh"
#include "../../nbo_correlatedgaussians_b200/csrc/necg_maps.h"

using namespace necg;

namespace {

const double kNaN = std::numeric_limits<double>::quiet_NaN();

struct Args {
    int n, nst, K;
    double efs;
    const double *mass, *ncv, *scvv, *sml, *sms;
};

// variant: 0 one-warp tiles, 1 with ket records re-read at each use, 2 staged ket
// records, 8 / 12 / 16 blocks of that many warps
template <int N> struct Pass {
    static constexpr int PB = SumFields<N>::size;
    Args a;
    Consts<N> cs;
    std::vector<int> pinv;
    bool ok;
    RawMapTable table;
    RawMap kmap;
    int variant, LC, npc;
    const double *C;
    std::vector<double> bra, ket, psym, xsym, sums;
    SymQueue q;
    SymLists lists;
    std::vector<int2> tiles, groups, urange, bgroups, burange;
    std::vector<int> start, tslot;
    int status[2] = {0, 0x7fffffff};

    Pass(const Args &args, const double *x, int variant_, int LC_, int npc_, int sms)
        : a(args), variant(variant_), LC(LC_), npc(variant_ >= 8 ? 1 : npc_) {
        const int K = a.K, nst = a.nst, nkb = row_blocks(K);
        ok = inverse_terms(N, nst, a.sml, a.sms, pinv);
        if (!ok) return;
        for (int i = 0; i < N * N; ++i) cs.M[i] = a.mass[i];
        for (int p = 1; p <= N; ++p)
            for (int r = 0; r < p; ++r) cs.cv[vidx(r, p)] = 2.0 * a.ncv[r] * a.ncv[p] / NECG_SQRT_PI;
        for (int i = 0; i < N; ++i) cs.q[i] = a.ncv[i + 1];
        cs.efs = a.efs;
        cs.sqrt8n = ::sqrt(::pow(8.0, N));
        table = raw_map_table(N, nst, a.sml, a.sms, KetSlots<N>::SL, [](int f) { return KetSlots<N>::slot(f); });
        kmap = RawMap{table.cnt.data(), table.src.data(), table.coef.data(), table.maxnz, table.fold};
        C = x + (size_t)K * (tri(N) + 3 * N);
        bra.assign((size_t)BraLayout<N>::size * 32 * nkb, kNaN);
        ket.assign((size_t)KetLayout<N>::size * K * nst + 2, kNaN);
        for (int k = 0; k < K; ++k) prep_bra_at<N>(x + (size_t)k * (tri(N) + 3 * N), cs, bra_at<N>(bra.data(), K, k), 32);
        for (int id = 0; id < K * nst; ++id)
            prep_ket_one<N>(x, C, nst, cs, a.sml, a.sms, a.scvv, kets(), id, pinv.data(), false);
        if (table.fold)  // general shift maps
            for (int id = 0; id < K * nst; ++id)
                prep_ket_one<N>(x, C, nst, cs, a.sml, a.sms, a.scvv, kets(), id, pinv.data(), true);
        q = sym_queue(K, LC, variant >= 8 ? variant : 8, nst, sms);
        tiles.resize(q.ntiles);
        tslot.resize(q.ntiles);
        groups.resize(q.units());
        urange.resize(nkb);
        burange.resize(nkb);
        start.resize(nkb + 1);
        bgroups.resize(groups_before(K, LC, 8, -1));
        lists = SymLists{tiles.data(), start.data(), groups.data(), urange.data(), tslot.data(), bgroups.data(), burange.data()};
        for (int kb = 0; kb < nkb; ++kb)
            for (int j = 0; j < 128; ++j) fill_sym_lists(q, lists, kb, j, 128);
        psym.assign((size_t)q.ntiles * PB * (32 + LC) * 2 * npc, kNaN);
        xsym.assign((size_t)q.ntail * q.w * (q.parts - 1) * fsym_tail_slot(PB, LC) + 1, kNaN);
    }
    double *kets() { return ket.data() + ((size_t)ket.data() / 8 & 1); }  // 16-byte records
    double *part_k() { return psym.data() + (size_t)q.ntiles * npc * 2 * PB * 32; }

    template <bool VKET, bool SKET, bool KE> void warp_tiles(double E, double *H, double *S, int t0, int t1) {
        const size_t KK = (size_t)a.K * a.K;
        std::vector<double> smem(2 * PB * 32 + ket_table<N>(2) + ket_red<N>() + 2 * KetLayout<N>::size + 2);
        for (int t = t0; t < t1; ++t)
            for (int pc = 0; pc < npc; ++pc) {
                std::fill(smem.begin(), smem.end(), kNaN);
                double *base = smem.data(), *sk = base + 2 * PB * 32 + ket_table<N>(2) + ket_red<N>();
                sk += (size_t)sk / 8 & 1;
                const FusedSmem sm{base, base + 2 * PB * 32, base + 2 * PB * 32 + ket_table<N>(2), sk};
                const int PC = (a.nst + npc - 1) / npc, p0 = std::min(pc * PC, a.nst), p1 = std::min(p0 + PC, a.nst);
                simt::run_block(32, [&] {
                    fsym_tile<N, VKET, false, SKET, true, KE>(t * npc + pc, tiles[t], LC, a.K, a.nst, cs, bra.data(), kets(),
                                                              C, kmap, H ? H + pc * KK : nullptr, H ? S + pc * KK : nullptr,
                                                              psym.data(), part_k(), status, sm, false, nullptr, p0, p1,
                                                              TileOut{}, E);
                });
            }
    }
    template <int W, bool KE> void block_units(double E, double *H, double *S) {
        std::vector<double> smem(fsym_block_smem_bytes<N>(W) / 8 + 2);
        for (int g = 0; g < q.units(); ++g) {
            std::fill(smem.begin(), smem.end(), kNaN);
            double *base = smem.data() + ((size_t)smem.data() / 8 & 1);
            simt::run_block(32 * W, [&] {
                fsym_group<N, W, KE>(g, groups[g], q.tail0, start.data(), LC, a.K, a.nst, cs, bra.data(), kets(), C, kmap, H,
                                     S, psym.data(), part_k(), status, xsym.data(), E, base);
            });
        }
        if (H && q.ntail)
            for (int j = 0; j < q.ntail; ++j)
                for (int w = 0; w < W; ++w)
                    simt::run_block(256, [&] {
                        fix_tail_tile<N>(groups[q.tail0 + j * q.parts], j, w, W, LC, a.K, xsym.data(), H, S);
                    });
    }
    template <bool KE> void pairs(double E, double *H, double *S, int t0, int t1) {
        switch (variant) {
        case 0: warp_tiles<KE, false, KE>(E, H, S, t0, t1); break;
        case 1: warp_tiles<true, false, KE>(E, H, S, t0, t1); break;
        case 2: warp_tiles<true, true, KE>(E, H, S, t0, t1); break;
        case 8: block_units<8, KE>(E, H, S); break;
        case 12: block_units<12, KE>(E, H, S); break;
        case 16: block_units<16, KE>(E, H, S); break;
        }
    }
    template <bool KE> void sum(int t0, int t1) {
        const bool blocks = variant >= 8, tail = blocks && q.ntail && q.parts >= 2;
        sums.assign((size_t)kSumSets * PB * a.K, kNaN);
        const PassParts p{start.data(), blocks ? urange.data() : nullptr, tail ? tslot.data() : nullptr, psym.data(), part_k(),
                          xsym.data(), LC, a.K, t0, t1, npc, q.parts};
        std::vector<double> red(4 * 8 * 32);
        for (int kb = 0; kb < row_blocks(a.K); ++kb)
            for (int f = 0; f < (KE ? PB - 1 : PB); ++f)
                simt::run_block(256, [&] { sum_partials<N, !KE>(p, kb, f, sums.data(), (double(*)[8][32])red.data()); });
    }
    // g and GRADC (own_e), or the gradient fields, from the sums
    bool finish(bool own_e, double E, double norm, bool ke, double *f, double *g, double *gradc, double *fields) {
        std::vector<double> smem(FinishSmem<N>::size), sh(64), en(4);
        bool fin = true;
        for (int kb = 0; kb < (a.K + 31) / 32; ++kb) {
            std::fill(smem.begin(), smem.end(), kNaN);
            simt::run_block(256, [&] {
                if (own_e) {
                    energy_from_rows<N>(sums.data(), C, a.K, (double(*)[32])sh.data(), en.data());
                    const int k = kb * 32 + threadIdx.x;
                    if (threadIdx.x < 32 && k < a.K) gradc[k] = gradc_from_rows<N>(sums.data(), a.K, k, en.data());
                }
                const double e = own_e ? en[0] : E, nrm = own_e ? en[1] : norm;
                if (!finish_block<N>(sums.data(), a.K, bra.data(), C, cs, kmap.fold, ke ? 0.0 : 2.0 * e, nrm, kb, fields, g,
                                     smem.data()))
                    fin = false;
            });
        }
        if (own_e && f) *f = en[0];
        return fin;
    }
};

int flags_of(const int *status, bool fin) { return status[0] | (fin ? 0 : 2); }

// mode 2: the fused evaluation; mode 1: the symmetric pass with the fused E.
template <int N>
int outprod(const Args &a, const double *x, int mode, int variant, int LC, int npc, int sms, double *f, double *g, double *H,
            double *S) {
    Pass<N> p(a, x, variant, LC, npc, sms);
    if (!p.ok) return -3;
    const size_t KK = (size_t)a.K * a.K, siv = (size_t)a.K * (tri(N) + 3 * N);
    std::vector<double> Hp(KK * p.npc, kNaN), Sp(KK * p.npc, kNaN);
    p.template pairs<false>(0.0, Hp.data(), Sp.data(), 0, p.q.ntiles);
    for (size_t i = 0; i < KK; ++i) {
        H[i] = Hp[i];
        S[i] = Sp[i];
        for (int pc = 1; pc < p.npc; ++pc) {
            H[i] += Hp[pc * KK + i];
            S[i] += Sp[pc * KK + i];
        }
    }
    p.template sum<false>(0, p.q.ntiles);
    bool fin = p.finish(true, 0.0, 0.0, false, f, g, g + siv, nullptr);
    if (mode == 2) return flags_of(p.status, fin);
    double cSc = 0.0;
    for (int i = 0; i < a.K; ++i)
        for (int j = 0; j < a.K; ++j) cSc += p.C[i] * S[(size_t)i * a.K + j] * p.C[j];
    Pass<N> s(a, x, variant, LC, 1, sms);
    s.template pairs<true>(*f, nullptr, nullptr, 0, s.q.ntiles);
    s.template sum<true>(0, s.q.ntiles);
    std::fill(g, g + siv, kNaN);
    fin = s.finish(false, *f, 1.0 / cSc, true, nullptr, g, nullptr, nullptr);
    return flags_of(s.status, fin);
}

// A rank's share: rows of H C and S C and the sums of tiles [t0, t1).
template <int N>
int shard_pairs(const Args &a, const double *x, int LC, int t0, int t1, double *rows, double *sums, int *ntiles) {
    Pass<N> p(a, x, 2, LC, 1, 148);
    if (!p.ok) return -3;
    *ntiles = p.q.ntiles;
    if (t0 < 0 || t1 > p.q.ntiles || t1 < t0) return -4;
    p.template pairs<false>(0.0, nullptr, nullptr, t0, t1);
    if (t1 > t0) p.template sum<false>(t0, t1);
    else p.sums.assign((size_t)kSumSets * Pass<N>::PB * a.K, 0.0);
    constexpr int PB = Pass<N>::PB, R = SumFields<N>::row;
    for (int i = 0; i < 2 * a.K; ++i) {  // rows_from_sums_kernel
        const int which = i >= a.K, m = i - which * a.K;
        rows[i] = p.sums[(size_t)(which * PB + R) * a.K + m] + p.sums[(size_t)((2 + which) * PB + R) * a.K + m];
    }
    std::copy(p.sums.begin(), p.sums.end(), sums);
    return p.status[0];
}

// Its gradient fields once E is known.
template <int N> int shard_fields(const Args &a, const double *x, const double *sums, double E, double norm, double *fields) {
    Pass<N> p(a, x, 2, 1, 1, 148);
    if (!p.ok) return -3;
    p.sums.assign(sums, sums + (size_t)kSumSets * Pass<N>::PB * a.K);
    p.finish(false, E, norm, false, nullptr, nullptr, nullptr, fields);
    return 0;
}

// GRADA from summed fields (grad_reduce_kernel).
template <int N> int shard_finish(const Args &a, const double *x, const double *fields, double norm, double *g) {
    Pass<N> p(a, x, 2, 1, 1, 148);
    int flags = 0;
    for (int k = 0; k < a.K; ++k)
        if (!grad_reduce_at<N>(fields, 1, a.K, bra_at<N>(p.bra.data(), a.K, k), 32, norm * p.C[k], g, k)) flags |= 2;
    return flags;
}

}  // namespace

#define DISPATCH(n, expr)                             \
    try {                                             \
        switch (n) {                                  \
        case 1: { constexpr int N = 1; return expr; } \
        case 2: { constexpr int N = 2; return expr; } \
        case 3: { constexpr int N = 3; return expr; } \
        case 4: { constexpr int N = 4; return expr; } \
        case 5: { constexpr int N = 5; return expr; } \
        default: return -2;                           \
        }                                             \
    } catch (const std::exception &e) {               \
        fprintf(stderr, "%s\n", e.what());            \
        return -9;                                    \
    }
#define PROBLEM                                                                                                      \
    int n, int nst, int K, double efs, const double *mass, const double *ncv, const double *scvv, const double *sml, \
        const double *sms
#define ARGS Args a{n, nst, K, efs, mass, ncv, scvv, sml, sms}

extern "C" int simt_outprod(PROBLEM, const double *x, int mode, int variant, int lc, int npc, int sm_count, double *f, double *g,
                            double *H, double *S) {
    ARGS;
    DISPATCH(n, (outprod<N>(a, x, mode, variant, lc, npc, sm_count, f, g, H, S)));
}
extern "C" int simt_shard_pairs(PROBLEM, const double *x, int lc, int t0, int t1, double *rows, double *sums, int *ntiles) {
    ARGS;
    DISPATCH(n, (shard_pairs<N>(a, x, lc, t0, t1, rows, sums, ntiles)));
}
extern "C" int simt_shard_fields(PROBLEM, const double *x, const double *sums, double E, double norm, double *fields) {
    ARGS;
    DISPATCH(n, (shard_fields<N>(a, x, sums, E, norm, fields)));
}
extern "C" int simt_shard_finish(PROBLEM, const double *x, const double *fields, double norm, double *g) {
    ARGS;
    DISPATCH(n, (shard_finish<N>(a, x, fields, norm, g)));
}
