// necg_device.cuh -- device-side pieces shared by the single-instance kernels
// (necg_kernels.cu) and the batched persistent kernels (necg_batch.cu): the
// shared-memory accumulators, the status word, and the body of one tile of the
// fused pass.
#pragma once
#include <cuda_runtime.h>

#include "necg_lanes.cuh"
#include "necg_math.cuh"
#include "necg_tiles.h"

namespace necg {

// Gradient accumulators of one lane in shared memory, interleaved by lane
// (field t of lane j at t * 32 + j): conflict-free, and not held in registers.
template <int N> struct SmemAcc {
    double *p;  // shared base + lane
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int t = 0; t < Part<N>::size; ++t) p[t * 32] = 0.0;
    }
    __device__ __forceinline__ double &g(int t) { return p[t * 32]; }
    __device__ __forceinline__ double &d() { return p[tri(N) * 32]; }
    __device__ __forceinline__ double &s(int t) { return p[(tri(N) + 1 + t) * 32]; }
};

// Stage the bra records' term fields of row block kb for BraSmem (by a block of
// `threads` threads; the caller synchronises).
template <int N>
__device__ __forceinline__ void stage_bras(double *sbra, const double *__restrict__ bra, int K, int kb, int threads) {
    const double *bk = bra + (size_t)kb * (BraLayout<N>::size * 32);
    const int first = kb == 0 ? row_pad(K) : 0;
    for (int i = threadIdx.x; i < BraLayout<N>::term * 32; i += threads) sbra[i] = bk[(i & ~31) + max(i & 31, first)];
}

// Copy a ket record of nd doubles (nd even: records are 16-byte multiples, at
// 16-byte aligned addresses) from global to shared memory without waiting:
// 16-byte cp.async per lane, one commit group per record.
__device__ __forceinline__ void ket_fetch(double *dst, const double *src, int nd, int lane) {
    for (int i = lane; 2 * i < nd; i += 32) {
#ifdef __CUDACC__
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + 2 * i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + 2 * i) : "memory");
#else
        simt::copy16(dst + 2 * i, src + 2 * i);
#endif
    }
#ifdef __CUDACC__
    asm volatile("cp.async.commit_group;" ::: "memory");
#endif
}
// Wait for this lane's copies and make the warp's copies visible to the warp.
__device__ __forceinline__ void ket_wait() {
#ifdef __CUDACC__
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#else
    simt::copies_wait();
#endif
    __syncwarp();
}

// Status word: [0] bit flags, [1] first failing pair (row-major k*K + l).
__device__ __forceinline__ void flag_status(int *status, int flags, int pair) {
    if (!flags) return;
    atomicOr(status, flags);
    atomicMin(status + 1, pair);
}

// Where a part of a split tile of the block variants writes instead of the
// main buffers (slot < 0: the main buffers): slot `slot` of x, fsym_tail_slot
// doubles holding its ket partials, then its LC x 64 H and S sums (H for the 32
// bras, then S).  The address is formed where it is used, so that
// it does not hold registers through the term loop.
struct TileOut {
    double *x = nullptr;
    int slot = -1;
};

// Doubles of a warp's ket tables (16 rows) in the fused pass (MATS = 2: H and S)
// or the symmetric pass (MATS = 1: the combined gradient).
template <int N> __host__ __device__ constexpr int ket_table(int mats) { return 16 * (mats * KetSlots<N>::SL + 1); }

// Doubles of the reduced ket fields of such a table: one per slot and lane.
template <int N> __host__ __device__ constexpr int ket_red() { return 2 * KetSlots<N>::SL > 32 ? 64 : 32; }

// Shared memory of one warp's tile: bra accumulators (2 * PB * 32 doubles), the
// ket table (ket_table) and the reduced ket fields (ket_red).  Sized by the caller
// for its largest n.
struct FusedSmem {
    double *sacc, *krow, *kred;
    double *sket;  // SKET: two ket-record buffers of this warp (16-byte aligned)
};

// term_raw's output in a tile: the bra's weighted raw values are added to the lane's
// accumulators, the ket's summed over lane pairs into the warp's table.  Lanes 2i and
// 2i+1 exchange one value per pair of fields: lane 2i keeps the first field, lane
// 2i+1 the second, each adds its partner's, and both store to row i (one
// select-and-shuffle per two fields, and half the rows to sum).
// KE (E known): the S fields go to the bra only, and H's are the combined ones.
template <int N, bool KE> struct TileOutput {
    using RP = RawPairs<N>;
    static constexpr bool kets = true, ket_s = !KE;
    static constexpr int PB = SumFields<N>::size, SL = KetSlots<N>::SL;
    double *acc;  // this lane's accumulators: H fields, then S fields, 32 doubles apart
    double *row;  // the lane pair's row, + 8 for the odd lane
    bool odd;
    double wb, wk, wob, wok;
    __device__ __forceinline__ void begin(double ov) {
        wob = wb * ov;
        wok = wk * ov;
    }
    __device__ __forceinline__ void bra(int f, double v) { acc[f * 32] = fma(wob, v, acc[f * 32]); }
    __device__ __forceinline__ double exchange(double va, double vb) {
        const double send = wok * (odd ? va : vb);
        return fma(wok, odd ? vb : va, __shfl_xor_sync(0xffffffffu, send, 1));
    }
    template <int I> __device__ __forceinline__ void sb(double va, double vb) {
        bra(PB + RP::fa(I), va);
        bra(PB + RP::fb(I), vb);
    }
    template <int I> __device__ __forceinline__ void hb(double va, double vb) {
        bra(RP::fa(I), va);
        bra(RP::fb(I), vb);
    }
    template <int I> __device__ __forceinline__ void sk(double va, double vb) {
        row[SL + KetSlots<N>::of_pair(I)] = exchange(va, vb);
    }
    template <int I> __device__ __forceinline__ void hk(double va, double vb) {
        row[KetSlots<N>::of_pair(I)] = exchange(va, vb);
    }
    __device__ __forceinline__ void scalar(double e2) {
        constexpr int p = KetSlots<N>::of_pair(RP::count - 1);
        bra(RP::scalar, e2);
        acc[(PB + RP::scalar) * 32] += wob;
        if (KE) {
            const double v = wok * e2;  // the odd lane's copy lands in an unused slot
            row[p] = v + __shfl_xor_sync(0xffffffffu, v, 1);
        } else {  // the even lane keeps H's scalar, the odd one S's
            const double vh = wok * e2, send = odd ? vh : wok;
            row[odd ? SL + p - 8 : p] = (odd ? wok : vh) + __shfl_xor_sync(0xffffffffu, send, 1);
        }
    }
    __device__ __forceinline__ void sb1(int, double) {}  // n = 6 has no symmetric passes
    __device__ __forceinline__ void hb1(int, double) {}
};

// One field of fold_raw at run time, from the reduced slots of one matrix.
template <int N>
__device__ __noinline__ double fold_slot(const double *slots, int f, const double *kr) {
    using KL = KetLayout<N>;
    constexpr int TR = tri(N);
    auto r = [&](int q) {
        double v = 0.0;
#pragma unroll
        for (int u = 0; u < Part<N>::size; ++u)
            if (u == q) v = slots[KetSlots<N>::slot(u)];
        return v;
    };
    if (f == TR) return 0.375 * r(TR);
    if (f < TR) return 0.5 * r(f);
    const int i = (f - TR - 1) / 3, c = (f - TR - 1) - 3 * i;
    double v = 0.0;
    for (int k = 0; k < N; ++k) v += kr[KL::Ap + (i >= k ? i * (i + 1) / 2 + k : k * (k + 1) / 2 + i)] * r(TR + 1 + 3 * k + c);
    return v;
}

// One tile of the pair passes over unordered pairs (k >= l).  Each term gives
// the raw values of term_raw (h, ov and their derivatives for the bra and for the
// ket); the bra's weighted sums stay in the lane's accumulators, the ket's are
// summed over the warp per (l, P), mapped to l's frame and summed over P.
//   !KE, the fused pass: H_kl = H_lk and S_kl are the sums over P of h and ov,
//        written when H is not null and always summed into the rows of H C and
//        S C (SumFields::row); the H and S fields are kept apart, since E is not
//        known until those rows are.
//   KE, the symmetric gradient pass (E = Egiven known): the combined gradient
//        of h - E ov, and the S fields for the bra only (its explicit share).
// Tile t = (kb, lc): the bras of row block kb, kets l in [lc LC, lc LC + LC).  Bra
// partials (PB = SumFields::size): part_b[((t * 2 + which) * PB + f) * 32 + lane];
// ket partials: part_k[((t * LC + l - l0) * 2 + which) * PB + f], which = 0 for H
// (or the combined gradient) and 1 for S (not written for the ket when KE).
//
// Shared memory per warp must stay under 228 KB / 8 for 8 resident warps, so the
// ket rows of two lanes are added before they are written (TileOutput) and the
// table has 16 rows.  The shuffles need the whole warp, so every lane evaluates a
// term: a lane without a pair (l > k, or no basis) evaluates the finite pair
// (l, l, P) with zero weights, which adds nothing.
// VKET: ket records re-read at each use (fewer live registers).
// idle: the warp has no tile (its accumulators are set to zero all the same).
// SBRA: the 32 bras of row block tl.x are staged in shared memory at sbra (field f
// of lane j at sbra[f * 32 + j]; lanes without a basis hold basis 0) and read there instead of from global memory.
// SKET: each (l, P) ket record is copied by the warp into one of its two
// buffers at sm.sket and read there; the copy of the next term's record
// (cp.async) runs while the current term is evaluated.
// [p0, p1): the symmetry terms this tile takes (p1 < 0: all nst).  A pass whose
// tiles split the terms writes each split's partials to its own slot (t is then
// the slot index) and each split's H, S sums to its own K x K buffer, or (xo)
// to the compact buffers of one part of a split tile.
// WB: write the bra partials to part_b (false: the caller reduces the warps'
// accumulators, left in sm.sacc, itself).
template <int N, bool VKET, bool SBRA = false, bool SKET = false, bool WB = true, bool KE = false>
__device__ __forceinline__ void fsym_tile(int t, int2 tl, int LC, int K, int nst, const Consts<N> &cs,
                                          const double *__restrict__ bra, const double *__restrict__ ket,
                                          const double *__restrict__ C, const RawMap &kmap,
                                          double *__restrict__ H, double *__restrict__ S,
                                          double *__restrict__ part_b, double *__restrict__ part_k,
                                          int *status, FusedSmem sm, bool idle = false,
                                          const double *sbra = nullptr, int p0 = 0, int p1 = -1,
                                          TileOut xo = TileOut{}, double Egiven = 0.0) {
    using KL = KetLayout<N>;
    constexpr int PS = Part<N>::size, PB = SumFields<N>::size, SL = KetSlots<N>::SL;
    constexpr int COLS = (KE ? 1 : 2) * SL;         // 16, 32 or 64 ket slots per row
    constexpr int STRIDE = COLS + 1;
    constexpr int NC = COLS > 32 ? 2 : 1;           // slots per lane
    static_assert(PS <= 32 && SL <= 32, "the symmetric passes need tri(n) + 1 + 3n <= 32");
    const int lane = threadIdx.x & 31;
    double *krow = sm.krow, *kred = sm.kred;
    const int k = tl.x * 32 + lane - row_pad(K);
    const int l0 = tl.y * LC;
    const int l1 = idle ? l0 : min(l0 + LC, row_last(K, tl.x) + 1);
    const bool kval = k >= 0 && !idle;
    const double Ck = kval ? C[k] : 0.0;
#pragma unroll
    for (int f = 0; f < 2 * PB; ++f) sm.sacc[f * 32 + lane] = 0.0;
    TileOutput<N, KE> out;
    out.acc = sm.sacc + lane;
    out.row = krow + (lane >> 1) * STRIDE + 8 * (lane & 1);
    out.odd = (lane & 1) != 0;
    const double E2 = KE ? 2.0 * Egiven : 0.0;
    // the slot this lane sums, maps and writes: js of matrix `which` (NC = 2: of both)
    const int js = lane & (SL - 1), which = NC == 2 ? 0 : lane / SL;
    int fld = -1;  // its field
#pragma unroll
    for (int f = 0; f < PS; ++f)
        if (KetSlots<N>::slot(f) == js) fld = f;
    const bool mine = fld >= 0 && lane < COLS;
    bool ok = true;
    int flags = 0, bad = 0x7fffffff;  // smallest failing pair (row-major k K + l)
    const int pend = p1 < 0 ? nst : p1;
    int cur = 0;  // SKET: the buffer that holds the current term's record
    if constexpr (SKET) {
        if (l0 < l1 && p0 < pend)
            ket_fetch(sm.sket, ket + ((size_t)l0 * nst + p0) * KL::size, KL::size, lane);
    }
    for (int l = l0; l < l1; ++l) {
        double ak[NC], hsum = 0.0, ssum = 0.0;
#pragma unroll
        for (int q = 0; q < NC; ++q) ak[q] = 0.0;
        const bool active = kval && l <= k;
        const BraRef b{bra_at<N>(bra, K, active ? k : l)};
        for (int P = p0; P < pend; ++P) {
            const double *kr = ket + ((size_t)l * nst + P) * KL::size;
            if constexpr (SKET) {
                ket_wait();  // this term's record is in buffer cur
                int nl = l, nP = P + 1;
                if (nP >= pend) {
                    nl = l + 1;
                    nP = p0;
                }
                if (nl < l1)
                    ket_fetch(sm.sket + (cur ^ 1) * KL::size, ket + ((size_t)nl * nst + nP) * KL::size, KL::size,
                              lane);
                kr = sm.sket + cur * KL::size;
                cur ^= 1;
            }
            out.wb = active ? kr[KL::wC] : 0.0;
            out.wk = active && l < k ? 2.0 * Ck * kr[KL::winv] : 0.0;
            double eta2, ov;
            bool tok;
            if constexpr (SBRA && SKET)
                tok = term_raw<N, double>(BraSmem{sbra + lane}, KetSmem{kr}, cs, E2, out, eta2, ov);
            else if constexpr (SBRA)
                tok = term_raw<N, double>(BraSmem{sbra + lane}, KetRefV{kr}, cs, E2, out, eta2, ov);
            else if constexpr (SKET)
                tok = term_raw<N, double>(b, KetSmem{kr}, cs, E2, out, eta2, ov);
            else if constexpr (VKET)
                tok = term_raw<N, double>(b, KetRefV{kr}, cs, E2, out, eta2, ov);
            else
                tok = term_raw<N, double>(b, kr, cs, E2, out, eta2, ov);
            if (active) {
                if (!tok && ok) {  // the first pair of this lane that is not positive definite
                    ok = false;
                    bad = min(bad, k * K + l);
                }
                if (!KE) {
                    const double wo = kr[KL::w] * ov;
                    hsum += wo * eta2;
                    ssum += wo;
                }
            }
            __syncwarp();
            // the 16 rows of the ket table, summed as trees (four dependent adds
            // instead of sixteen), then mapped to l's frame
            {
                double v[NC][16];
#pragma unroll
                for (int r = 0; r < 16; ++r)
#pragma unroll
                    for (int q = 0; q < NC; ++q) v[q][r] = krow[r * STRIDE + 32 * q + (COLS < 32 ? lane & (COLS - 1) : lane)];
#pragma unroll
                for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
                    for (int r = 0; r < w; ++r)
#pragma unroll
                        for (int q = 0; q < NC; ++q) v[q][r] += v[q][r + w];
#pragma unroll
                for (int q = 0; q < NC; ++q) kred[32 * q + lane] = v[q][0];
            }
            __syncwarp();
            if (kmap.fold) {  // gradients in P's frame instead of raw sums
                const double *krg = ket + ((size_t)l * nst + P) * KL::size;
                double v[NC];
#pragma unroll
                for (int q = 0; q < NC; ++q) {
                    const int wq = which + q;
                    v[q] = mine ? fold_slot<N>(kred + wq * SL, fld, krg) : 0.0;
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < NC; ++q) kred[32 * q + lane] = v[q];
                __syncwarp();
            }
            if (mine) {
                const int e = P * SL + js, n = kmap.cnt[e];
                double m[NC];
#pragma unroll
                for (int q = 0; q < NC; ++q) m[q] = 0.0;
                for (int i = 0; i < n; ++i) {
                    const double c = kmap.coef[(size_t)e * kmap.maxnz + i];
                    const int s = kmap.src[(size_t)e * kmap.maxnz + i];
#pragma unroll
                    for (int q = 0; q < NC; ++q) m[q] += c * kred[(which + q) * SL + s];
                }
#pragma unroll
                for (int q = 0; q < NC; ++q) ak[q] += m[q];
            }
            __syncwarp();
        }
        double *pk = xo.slot >= 0 ? xo.x + (size_t)xo.slot * fsym_tail_slot(PB, LC) + (size_t)(l - l0) * 2 * PB
                                  : part_k + ((size_t)t * LC + (l - l0)) * 2 * PB;
        if (!KE) {
            hsum *= 0.5;
            if (active) {
                if (!isfinite(hsum) || !isfinite(ssum)) {
                    bad = min(bad, k * K + l);
                    flags |= 2;
                }
                if (H) {
                    if (xo.slot >= 0) {
                        double *hs = xo.x + (size_t)xo.slot * fsym_tail_slot(PB, LC) + (size_t)LC * 2 * PB;
                        hs[(l - l0) * 64 + lane] = hsum;
                        hs[(l - l0) * 64 + 32 + lane] = ssum;
                    } else {
                        H[(size_t)k * K + l] = hsum;
                        H[(size_t)l * K + k] = hsum;
                        S[(size_t)k * K + l] = ssum;
                        S[(size_t)l * K + k] = ssum;
                    }
                }
                const double Cl = C[l];
                out.acc[PS * 32] += hsum * Cl;
                out.acc[(PB + PS) * 32] += ssum * Cl;
            }
            // the ket's row: sum over the bras k > l (lane 0 ends with H's, lane 1 with S's)
            const double ch = active && l < k ? hsum * Ck : 0.0, cs_ = active && l < k ? ssum * Ck : 0.0;
            double r = (lane & 1 ? cs_ : ch) + __shfl_xor_sync(0xffffffffu, lane & 1 ? ch : cs_, 1);
#pragma unroll
            for (int o = 2; o < 32; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
            if (lane < 2) pk[lane * PB + PS] = r;
        }
        if (mine)
#pragma unroll
            for (int q = 0; q < NC; ++q) pk[(which + q) * PB + fld] = ak[q];
    }
    if (WB && kval) {
        double *pb = part_b + (size_t)t * 2 * PB * 32;
#pragma unroll
        for (int f = 0; f < 2 * PB; ++f) pb[f * 32 + lane] = sm.sacc[f * 32 + lane];
    }
    if (!ok) flags |= 1;
    flag_status(status, flags, bad);
    __syncwarp();
}

// Dynamic shared memory of a block of warps (doubles, 16-byte aligned): per warp its
// tile's areas (FusedSmem), then the bras that the warps share.
template <int N> __host__ __device__ constexpr int fsym_warp_smem() {
    return 2 * SumFields<N>::size * 32 + ket_table<N>(2) + ket_red<N>() + 2 * KetLayout<N>::size;
}
template <int N> __host__ __device__ constexpr int fsym_block_smem_bytes(int warps) {
    return (warps * fsym_warp_smem<N>() + BraLayout<N>::term * 32) * 8;
}

// One unit of a queue of tile groups by a block of WARPS warps: unit g = row block
// kb and ket chunks lc0 .. lc0 + WARPS - 1 (or one part of their symmetry terms),
// one per warp.  The unit's bras are staged in shared memory once for all warps, each
// warp stages its ket records, and the warps meet only at the unit's ends.  Parts
// after the first of a split group write to their own slots in xsym (groups split
// from unit tail0 on); KE: the symmetric pass with E known.
template <int N, int WARPS, bool KE>
__device__ __forceinline__ void fsym_group(int g, int2 gr, int tail0, const int *__restrict__ tstart, int LC, int K,
                                           int nst, const Consts<N> &cs, const double *__restrict__ bra,
                                           const double *__restrict__ ket, const double *__restrict__ C,
                                           const RawMap &kmap, double *__restrict__ H, double *__restrict__ S,
                                           double *__restrict__ part_b, double *__restrict__ part_k, int *status,
                                           double *__restrict__ xsym, double E, double *smem) {
    constexpr int PB = SumFields<N>::size, PER_WARP = fsym_warp_smem<N>(), TBL = ket_table<N>(2);
    const int w = threadIdx.x >> 5;
    double *base = smem + w * PER_WARP;
    double *sbra = smem + WARPS * PER_WARP;  // after the warps' areas
    const FusedSmem sm{base, base + 2 * PB * 32, base + 2 * PB * 32 + TBL, base + 2 * PB * 32 + TBL + ket_red<N>()};
    const int kb = gr.x, lc = sgroup_lc0(gr) + w;
    const bool idle = lc * LC > row_last(K, kb);  // past this block's triangle
    const int part = sgroup_part(gr), parts = sgroup_parts(gr);
    const int p0 = part * nst / parts, p1 = (part + 1) * nst / parts;  // balanced ranges
    TileOut xo;
    if (part > 0) {
        xo.x = xsym;
        xo.slot = (((g - tail0) / parts) * WARPS + w) * (parts - 1) + (part - 1);
    }
    stage_bras<N>(sbra, bra, K, kb, 32 * WARPS);
    __syncthreads();
    fsym_tile<N, true, true, true, false, KE>(tstart[kb] + lc, make_int2(kb, lc), LC, K, nst, cs, bra, ket, C, kmap,
                                              H, S, part_b, part_k, status, sm, idle, sbra, p0, p1, xo, E);
    // the unit's bra partials: its warps share the 32 bras, so their accumulators
    // are summed (in warp order) and written once, to the slot of unit g
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * PB * 32; i += 32 * WARPS) {
        if (kb == 0 && (i & 31) < row_pad(K)) continue;  // no basis
        double v = smem[i];
#pragma unroll
        for (int q = 1; q < WARPS; ++q) v += smem[q * PER_WARP + i];
        part_b[(size_t)g * 2 * PB * 32 + i] = v;
    }
    __syncthreads();  // sbra and the warps' areas are rewritten for the next unit
}

// H and S of one tile (warp w) of tail group j, when the caller wants them: add parts
// 1 .. parts - 1 (their slots in xsym, in part order) to what part 0 wrote, by a block
// of any size.  Entries that no part wrote (kets past K or above the diagonal, tiles
// past the block's triangle) are left alone.
template <int N>
__device__ __forceinline__ void fix_tail_tile(int2 gr, int j, int w, int W, int LC, int K, const double *__restrict__ xsym,
                                              double *__restrict__ H, double *__restrict__ S) {
    constexpr int PB = SumFields<N>::size;
    const int parts = sgroup_parts(gr), kb = gr.x, lc = sgroup_lc0(gr) + w;
    if (lc * LC > row_last(K, kb)) return;
    const size_t XS = fsym_tail_slot(PB, LC);
    const double *x0 = xsym + (size_t)(j * W + w) * (parts - 1) * XS + (size_t)LC * 2 * PB;
    for (int i = threadIdx.x; i < LC * 64; i += blockDim.x) {
        const int l = lc * LC + i / 64, r = i & 63, k = kb * 32 + (r & 31) - row_pad(K);
        if (k < 0 || l > k) continue;
        double *M = r < 32 ? H : S;
        double v = M[(size_t)k * K + l];
        for (int q = 0; q < parts - 1; ++q) v += x0[q * XS + i];
        M[(size_t)k * K + l] = v;
        M[(size_t)l * K + k] = v;
    }
}

// Where the partials of a symmetric pass are and which of them count: tiles
// [t0, t1) (a shard of the pass) of the tile list whose row blocks start at
// tstart.  Bra partials: tile t's splits are slots t npc .. t npc + npc - 1, or
// (urange: the block variants) row block kb's are the queue units urange[kb].
// Ket partials: the tile's splits likewise and, for a tile of a split group
// (tslot[t] >= 0), slots tslot[t] .. + parts - 2 of xsym.
struct PassParts {
    const int *tstart;
    const int2 *urange;
    const int *tslot;
    const double *part_b, *part_k, *xsym;
    int LC, K, t0, t1, npc, parts;
};

// One block of 256 threads sums field f of the 32 bases of row block kb: their
// bra partials come from every tile of the block (up to K / LC of them), their
// ket partials from one tile per later row block, so the 8 warps take every 8th
// of each and their sums are combined in a fixed order.  Into sums (kSumSets
// sets); TWO: the ket has S partials too.
template <int N, bool TWO>
__device__ __forceinline__ void sum_partials(const PassParts &p, int kb, int f, double *__restrict__ sums,
                                             double (*red)[8][32]) {
    constexpr int PB = SumFields<N>::size;
    const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
    const int K = p.K, LC = p.LC, m = kb * 32 + lane - row_pad(K);
    const int ta = p.urange ? p.urange[kb].x : max(p.tstart[kb], p.t0) * p.npc;
    const int tb = p.urange ? p.urange[kb].y : min(p.tstart[kb + 1], p.t1) * p.npc;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int t = ta + seg; t < tb; t += 8) {
        v[0] += p.part_b[(((size_t)t * 2 + 0) * PB + f) * 32 + lane];
        v[1] += p.part_b[(((size_t)t * 2 + 1) * PB + f) * 32 + lane];
    }
    if (m >= 0) {
        const int lc = m / LC, ll = m - lc * LC;
        const int nkb = row_blocks(K);
        int kb0 = m + row_pad(K) - 31;  // first row block that meets ket m
        kb0 = kb0 > 0 ? (kb0 + 31) >> 5 : 0;
        for (int q = kb0 + seg; q < nkb; q += 8) {
            const int t = p.tstart[q] + lc;
            if (t < p.t0 || t >= p.t1) continue;
            for (int pc = 0; pc < p.npc; ++pc) {
                const double *pk = p.part_k + ((size_t)(t * p.npc + pc) * LC + ll) * 2 * PB + f;
                v[2] += pk[0];
                if (TWO) v[3] += pk[PB];
            }
            if (p.tslot && p.tslot[t] >= 0)
                for (int pc = 0; pc < p.parts - 1; ++pc) {
                    const double *pk = p.xsym + (size_t)(p.tslot[t] + pc) * fsym_tail_slot(PB, LC) + (size_t)ll * 2 * PB + f;
                    v[2] += pk[0];
                    if (TWO) v[3] += pk[PB];
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) red[i][seg][lane] = v[i];
    __syncthreads();
    if (seg < 4 && m >= 0) {  // warp i: set i
        double s = red[seg][0][lane];
#pragma unroll
        for (int q = 1; q < 8; ++q) s += red[seg][q][lane];
        sums[((size_t)seg * PB + f) * K + m] = s;
    }
    __syncthreads();
}

// E = C^T H C / C^T S C and norm = 1 / C^T S C (python/outprod.py:65-68) from the
// row sums, by every thread of the block in the same fixed order; en = {E, norm,
// cHc, cSc} in shared memory, sh: 2 x 32 doubles.
template <int N>
__device__ __forceinline__ void energy_from_rows(const double *__restrict__ sums, const double *__restrict__ C, int K,
                                                 double (*sh)[32], double *en) {
    constexpr int PB = SumFields<N>::size, R = SumFields<N>::row;
    double ah = 0.0, as = 0.0;
    for (int i = threadIdx.x; i < K; i += blockDim.x) {
        const double c = C[i];
        ah += c * (sums[(size_t)R * K + i] + sums[(size_t)(2 * PB + R) * K + i]);
        as += c * (sums[(size_t)(PB + R) * K + i] + sums[(size_t)(3 * PB + R) * K + i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ah += __shfl_xor_sync(0xffffffffu, ah, o);
        as += __shfl_xor_sync(0xffffffffu, as, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = ah;
        sh[1][threadIdx.x >> 5] = as;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double th = 0.0, ts = 0.0;
        for (int j = 0; j < (int)(blockDim.x >> 5); ++j) {
            th += sh[0][j];
            ts += sh[1][j];
        }
        en[0] = th / ts;
        en[1] = 1.0 / ts;
        en[2] = th;
        en[3] = ts;
    }
    __syncthreads();
}

// Shared memory of finish_block (doubles).
template <int N> struct FinishSmem {
    static constexpr int PS = Part<N>::size, blk = tri(N) + 3 * N;
    static constexpr int r = 0;                    // combined raw sums, then the gradient fields
    static constexpr int s = r + PS * 32;          // the bra's S sums, then the output
    static constexpr int out = s;                  // blk x 32, basis-major with an odd stride (<= PS)
    static constexpr int rec = s + PS * 32;        // A and L of the 32 bases
    static constexpr int y = rec + 2 * tri(N) * 32;
    static constexpr int MA = y + 3 * N * 32;
    static constexpr int size = MA + N * N * 32;
    static_assert((blk | 1) <= PS, "the output fits where the S sums were");
    // more than 48 KB would need the opt-in and another split of the SM's L1 (n = 5
    // took 61 KB with areas of their own: 10 us more per evaluation at any K)
    static_assert(N > 5 || size * 8 <= 48 * 1024, "shared memory");
};

// The gradients of the bases 32 kb .. 32 kb + 31 from their per-basis sums, by one
// block of 256 threads: every step is split over the warps by matrix row, lane =
// basis, so that the loads of all fields are in flight at once and no thread
// walks the whole chain (one thread per basis took 11 us at n = 5 for any K).  E2 =
// 2 E, or 0 where the sums are combined already (no S set of the ket then).  The
// bra's explicit share of tau (explicit_tau), the fold (fold_raw) and the map to
// vech(L) (a_to_vech) as there, row by row.  GRADA (scaled by norm C_k) goes to g,
// or the gradient fields, field-major, to `fields`.  Returns whether this
// thread's outputs are finite.
template <int N>
__device__ __forceinline__ bool finish_block(const double *__restrict__ sums, int K, const double *__restrict__ bra,
                                             const double *__restrict__ C, const Consts<N> &cs, int folded, double E2,
                                             double norm, int kb, double *__restrict__ fields,
                                             double *__restrict__ g, double *sm) {
    using BL = BraLayout<N>;
    using FS = FinishSmem<N>;
    constexpr int TR = tri(N), PS = Part<N>::size, PB = SumFields<N>::size, blk = FS::blk;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = min(kb * 32 + lane, K - 1);
    const int nk = min(32, K - kb * 32);
    constexpr int A = FS::rec, L = A + TR * 32;
    const double *bk = bra_at<N>(bra, K, k);
    auto ket = [&](int f) {  // the kets' combined sum (folded: their gradient)
        const double *q = sums + (size_t)(2 * PB + f) * K + k;
        return E2 != 0.0 ? q[0] - E2 * q[(size_t)PB * K] : q[0];
    };
#pragma unroll
    for (int f = w; f < PS; f += 8) {
        const double *q = sums + (size_t)f * K + k;
        const size_t set = (size_t)PB * K;
        double r = q[0];
        const double bs = q[set];
        if (E2 != 0.0) r -= E2 * bs;
        sm[FS::r + f * 32 + lane] = folded ? r : r + ket(f);
        sm[FS::s + f * 32 + lane] = bs;
    }
#pragma unroll
    for (int f = w; f < TR; f += 8) {
        sm[A + f * 32 + lane] = bk[(BL::A + f) * 32];
        sm[L + f * 32 + lane] = bk[(BL::L + f) * 32];
    }
    __syncthreads();
    auto at = [&](int base, int f) -> double & { return sm[base + f * 32 + lane]; };
    const int i = w;  // this warp's matrix row
    if (i < N) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < N; ++q) v += at(A, sx(i, q)) * at(FS::s, TR + 1 + 3 * q + c);
            at(FS::y, 3 * i + c) = v;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < N; ++q) v += cs.M[i * N + q] * at(A, sx(q, j));
            at(FS::MA, i * N + j) = v;
        }
    }
    __syncthreads();
    if (i < N) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < N; ++q) v += cs.M[i * N + q] * at(FS::y, 3 * q + c);
            at(FS::r, TR + 1 + 3 * i + c) += 8.0 * v;
        }
        for (int j = 0; j <= i; ++j) {
            double v = 3.0 * cs.M[i * N + j] * at(FS::s, TR);
#pragma unroll
            for (int q = 0; q < N; ++q)
                v += 2.0 * (at(FS::MA, i * N + q) * at(FS::s, sx(q, j)) + at(FS::s, sx(i, q)) * at(FS::MA, j * N + q));
            at(FS::r, sx(i, j)) += 4.0 * v;
        }
    }
    __syncthreads();
    // the fold: matrix row i (in place: entry (i, j) reads only itself) and dF/ds row i
    const double F = 0.5 * at(FS::r, TR);
    double gs[3];
    if (i < N) {
        for (int j = 0; j <= i; ++j) {
            const double v = 0.5 * at(FS::r, sx(i, j));
            at(FS::r, sx(i, j)) = folded ? v + ket(sx(i, j)) : v;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = at(A, sx(i, 0)) * at(FS::r, TR + 1 + c);
#pragma unroll
            for (int q = 1; q < N; ++q) v += at(A, sx(i, q)) * at(FS::r, TR + 1 + 3 * q + c);
            gs[c] = folded ? v + ket(TR + 1 + 3 * i + c) : v;
        }
    }
    const double D = folded ? 0.75 * F + ket(TR) : 0.75 * F;
    __syncthreads();
    bool fin = true;
    if (fields) {
        if (i < N) {
#pragma unroll
            for (int c = 0; c < 3; ++c) at(FS::r, TR + 1 + 3 * i + c) = gs[c];
        }
        if (w == 0) at(FS::r, TR) = D;
        __syncthreads();
        if (lane < nk)
            for (int f = w; f < PS; f += 8) fields[(size_t)f * K + k] = at(FS::r, f);
    } else {
        const double sc = norm * C[k];
        double *o = sm + FS::out + lane * (blk | 1);
        if (i < N) {  // column i of vech(dF/dL): rows a = i .. N - 1
            const int j = i;
            int idx = j * N - j * (j - 1) / 2;
            for (int a = j; a < N; ++a) {
                double v = 0.0;
                for (int q = j; q < N; ++q) v += at(FS::r, sx(a, q)) * at(L, sx(q, j));
                v *= 2.0;
                if (a == j) v += 2.0 * D / at(L, sx(j, j));
                v *= sc;
                fin = fin && isfinite(v);
                o[idx++] = v;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double v = sc * gs[c];
                fin = fin && isfinite(v);
                o[TR + 3 * i + c] = v;
            }
        }
        __syncthreads();
        // the 32 blocks of g are contiguous
        for (int q = threadIdx.x; q < nk * blk; q += 256)
            g[(size_t)kb * 32 * blk + q] = sm[FS::out + (q / blk) * (blk | 1) + q % blk];
    }
    __syncthreads();
    return fin || lane >= nk;
}

// GRADC of basis i: 2 norm (H C - E S C)_i (python/make_grad.py:85).
template <int N>
__device__ __forceinline__ double gradc_from_rows(const double *__restrict__ sums, int K, int i, const double *en) {
    constexpr int PB = SumFields<N>::size, R = SumFields<N>::row;
    return 2.0 * en[1] * ((sums[(size_t)R * K + i] + sums[(size_t)(2 * PB + R) * K + i]) -
                          en[0] * (sums[(size_t)(PB + R) * K + i] + sums[(size_t)(3 * PB + R) * K + i]));
}

}  // namespace necg
