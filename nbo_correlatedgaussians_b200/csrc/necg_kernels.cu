// necg_kernels.cu -- sm_100a FP64 kernels of the ECG energy+gradient path.
//
// One outprod evaluation (python/outprod.py:20-76 + python/make_grad.py:18-90)
// is, with separate passes for the matrices and the gradient, the launch sequence
//   prep        per basis k:     A_k, S_k, A_k S_k, A_k M A_k, i1, |L_k|^{3/2}
//               per (l, P):      A_l' = P^T A_l P, S_l' = sms s_l and derived data
//   energy      triangle tiles:  H_kl, S_kl for k >= l  (the matel loop)
//   rows        per row:         (H C)_i, (S C)_i
//   finalize    one block:       E = C^T H C / C^T S C, norm, GRADC
//   grad        square tiles:    sum over (l, P) of the bra gradient of
//                                2 C_l w_P (h - E ov)    (the gradel loop)
//   grad_reduce per basis k:     sum the tile partials, map A-space to vech(L)
// and with the fused pass (unordered pairs)
//   prep, fsym  triangle tiles:  H and S sums and both gradients as raw sums
//   fsym_sum    per (32 bases, field): the tile partials
//   fsym_finish per basis k:     E, norm, GRADC from the row sums; gradient, vech(L)
// Tiles are one warp wide: lane = bra basis function k, while the ket (l, P)
// loops are warp-uniform, so ket records are read once per warp as broadcasts.
// The per-thread bodies live in necg_lanes.cuh.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include "necg_device.cuh"
#include "necg_kernels.cuh"
#include "necg_lanes.cuh"
#include "necg_math.cuh"

namespace necg {

// Ket records in device memory, read warp-uniformly.
struct DevKet {
    const double *p;
    __device__ __forceinline__ const double *at(size_t off) const { return p + off; }
};

// Bra records (the first nbb blocks) and ket records (the others), in one launch
// with the reset of the status words and of the block variants' queue head.
template <int N>
__global__ void __launch_bounds__(64) prep_kernel(const double *__restrict__ iv, const double *__restrict__ C, int K,
                                                  int nst, int nbb, Consts<N> cs, const double *__restrict__ sml,
                                                  const double *__restrict__ sms, const double *__restrict__ scvv,
                                                  const int *__restrict__ pinv, int general,
                                                  double *__restrict__ bra, double *__restrict__ ket, int *status,
                                                  int *qcount) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        status[0] = 0;
        status[1] = 0x7fffffff;
        if (qcount) *qcount = 0;
    }
    if ((int)blockIdx.x < nbb) {
        const int k = blockIdx.x * blockDim.x + threadIdx.x;
        if (k < K) prep_bra_at<N>(iv + (size_t)k * (tri(N) + 3 * N), cs, bra_at<N>(bra, K, k), 32);
        return;
    }
    const int id = (blockIdx.x - nbb) * blockDim.x + threadIdx.x;
    if (id < K * nst) prep_ket_one<N>(iv, C, nst, cs, sml, sms, scvv, ket, id, pinv, general);
}

// The tile lists: block kb writes row block kb's entries.  A few microseconds, once
// per size and setting.
__global__ void __launch_bounds__(128) tile_list_kernel(int2 *tiles, int K, int LC) {
    const int kb = blockIdx.x, t0 = tiles_before(K, LC, kb), nt = block_tiles(K, LC, kb);
    for (int lc = threadIdx.x; lc < nt; lc += blockDim.x) tiles[t0 + lc] = make_int2(kb, lc);
}
__global__ void __launch_bounds__(128) sym_lists_kernel(SymQueue q, SymLists o) {
    fill_sym_lists(q, o, blockIdx.x, threadIdx.x, blockDim.x);
}

// Energy tiles over the lower triangle (the loop of python/outprod.py:49-54 and
// python/necg.py:43-50), in the order of tile_list_kernel.
// One warp per block; MINW = minimum resident warps per SM the kernel is
// compiled for (register budget 65536 / (32 MINW) per thread).
template <int N, int MINW>
__global__ void __launch_bounds__(32, MINW) energy_kernel(const int2 *__restrict__ tiles, int ntiles,
                                                     int LC, int K, int nst, Consts<N> cs,
                                                     const double *__restrict__ bra,
                                                     const double *__restrict__ ket,
                                                     double *__restrict__ H, double *__restrict__ S,
                                                     double *__restrict__ Kin,
                                                     double *__restrict__ Pot, int *status) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= ntiles) return;
    const int2 tl = tiles[warp];
    int k, l0, lend;
    if (!energy_lane_range(tl.x, tl.y, lane, LC, K, k, l0, lend)) return;
    int bad = 0;
    const int fl = energy_lane<N, double>(BraRef{bra_at<N>(bra, K, k)}, DevKet{ket}, k, l0, lend, K, nst,
                                          cs, H, S, Kin, Pot, bad);
    flag_status(status, fl, bad);
}

// The same with W warps per tile, each over its share of the symmetry terms, for
// bases with too few tiles to fill the GPU (a tile is a chain of LC nst terms):
// the warps' sums of a pair meet in shared memory and are added in warp order.
// FP64 latency bounds it.  LiH K = 301 with H, S, Kinetic and Potential on a
// B200: 222 us one warp per tile (with an earlier term), 154 us with 2.
template <int N, int W>
__global__ void __launch_bounds__(32 * W) energy_split_kernel(const int2 *__restrict__ tiles, int LC, int K, int nst,
                                                              Consts<N> cs, const double *__restrict__ bra,
                                                              const double *__restrict__ ket,
                                                              double *__restrict__ H, double *__restrict__ S,
                                                              double *__restrict__ Kin, double *__restrict__ Pot,
                                                              int *status) {
    __shared__ double red[W][4][32];
    __shared__ int bad[W][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 tl = tiles[blockIdx.x];
    int k, l0, lend;
    const bool mine = energy_lane_range(tl.x, tl.y, lane, LC, K, k, l0, lend);
    const BraRef b{bra_at<N>(bra, K, mine ? k : 0)};
    const int p0 = w * nst / W, p1 = (w + 1) * nst / W;
    int flags = 0, pair = 0x7fffffff;
    for (int l = tl.y * LC; l < min(tl.y * LC + LC, K); ++l) {
        const bool has = mine && l < lend;
        if (has) {
            double sum[4];
            bad[w][lane] = !energy_sums<N, double>(b, DevKet{ket}, l, nst, p0, p1, cs, sum);
#pragma unroll
            for (int i = 0; i < 4; ++i) red[w][i][lane] = sum[i];
        }
        __syncthreads();
        if (w == 0 && has) {
            double v[4];
            bool ok = !bad[0][lane];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = red[0][i][lane];
            for (int q = 1; q < W; ++q) {
                ok = ok && !bad[q][lane];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] += red[q][i][lane];
            }
            const int fl = energy_store(v, ok, k, l, K, H, S, Kin, Pot);
            if (fl && !flags) pair = k * K + l;
            flags |= fl;
        }
        __syncthreads();
    }
    flag_status(status, flags, pair);
}

// rows[i] = (H C)_i, rows[K + i] = (S C)_i ; one warp per row.  Memory bound (16
// K^2 bytes); eight loads of each matrix in flight per lane (K = 2048 on a B200:
// 26 us with one, 22 us with eight).
__global__ void __launch_bounds__(256) rows_kernel(const double *__restrict__ H,
                                                   const double *__restrict__ S,
                                                   const double *__restrict__ C, int K,
                                                   double *__restrict__ rows) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= K) return;
    const double *h = H + (size_t)warp * K;
    const double *s = S + (size_t)warp * K;
    double ah = 0.0, as = 0.0;
    int j = lane;
    for (; j + 7 * 32 < K; j += 8 * 32) {
        double a[8], b[8], c[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            a[q] = h[j + 32 * q];
            b[q] = s[j + 32 * q];
            c[q] = C[j + 32 * q];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            ah += a[q] * c[q];
            as += b[q] * c[q];
        }
    }
    for (; j < K; j += 32) {
        const double c = C[j];
        ah += h[j] * c;
        as += s[j] * c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ah += __shfl_xor_sync(0xffffffffu, ah, o);
        as += __shfl_xor_sync(0xffffffffu, as, o);
    }
    if (lane == 0) {
        rows[warp] = ah;
        rows[K + warp] = as;
    }
}

// E = C^T H C / C^T S C, norm = 1 / C^T S C (python/outprod.py:65-68) and
// GRADC = 2 norm (H - E S) C (python/make_grad.py:85) into gradc[0 .. K).
// scal = {E, norm, cHc, cSc}.  With `given`, E and norm are the caller's
// (make_grad(eng, norm) semantics).  One block of 1024 threads; fixed-order tree.
__global__ void __launch_bounds__(1024) finalize_kernel(const double *__restrict__ rows,
                                                        const double *__restrict__ C, int K,
                                                        double *__restrict__ scal,
                                                        double *__restrict__ f_out,
                                                        double *__restrict__ gradc, int *status,
                                                        int given, double eng, double gnorm,
                                                        const double *__restrict__ given_dev,
                                                        double *__restrict__ en_out) {
    __shared__ double sh[2][32];
    double ah = 0.0, as = 0.0;
    for (int i = threadIdx.x; i < K; i += blockDim.x) {
        ah += C[i] * rows[i];
        as += C[i] * rows[K + i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ah += __shfl_xor_sync(0xffffffffu, ah, o);
        as += __shfl_xor_sync(0xffffffffu, as, o);
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        sh[0][w] = ah;
        sh[1][w] = as;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        ah = lane < nw ? sh[0][lane] : 0.0;
        as = lane < nw ? sh[1][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ah += __shfl_xor_sync(0xffffffffu, ah, o);
            as += __shfl_xor_sync(0xffffffffu, as, o);
        }
        if (lane == 0) {
            double E = ah / as, nrm = 1.0 / as;
            if (given == 1) {
                E = eng;
                nrm = gnorm;
            } else if (given == 2) {
                E = given_dev[0];
                nrm = given_dev[1];
            }
            scal[0] = E;
            scal[1] = nrm;
            scal[2] = ah;
            scal[3] = as;
            if (f_out) *f_out = E;
            if (en_out) {
                en_out[0] = E;
                en_out[1] = nrm;
            }
            if (!isfinite(E)) atomicOr(status, 2);
        }
    }
    __syncthreads();
    if (gradc) {
        const double E = scal[0], norm = scal[1];
        for (int i = threadIdx.x; i < K; i += blockDim.x)
            gradc[i] = 2.0 * norm * (rows[i] - E * rows[K + i]);
    }
}

// Gradient tiles over the full square of ordered pairs (the loop of
// python/make_grad.py:37-55, contracted with C on the fly as lines 61-79 do).
// Tile t = (kb, lc); lane k accumulates over l in the chunk and all P (raw H and
// S sums in shared memory) and writes its gradient to part[(lc * Part::size + f) * K + k].
template <int N, int MINW>
__global__ void __launch_bounds__(32, MINW) grad_kernel(int nkb, int nlc, int LC, int K, int nst,
                                                   Consts<N> cs, const double *__restrict__ bra,
                                                   const double *__restrict__ ket,
                                                   const double *__restrict__ scal, double lam,
                                                   double *__restrict__ part, int *status) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nkb * nlc) return;
    int k, lc, l0, l1;
    if (!grad_lane_range(warp, lane, nkb, LC, K, k, lc, l0, l1)) return;
    double *out = part + (size_t)lc * Part<N>::size * K + k;
    __shared__ double sacc[2 * Part<N>::size * 32];
    SmemAcc<N> accH{sacc + lane}, accS{sacc + Part<N>::size * 32 + lane};
    const bool ok = grad_lane<N, double>(BraRef{bra_at<N>(bra, K, k)}, DevKet{ket}, l0, l1, nst, cs, lam, scal[0],
                                         out, (size_t)K, accH, accS);
    if (!ok) flag_status(status, 1, k * K + l0);
}

// Symmetric gradient pass (E = scal[0] known; python/make_grad.py's role when H
// and S are given): each unordered pair (k >= l) once, bra and ket gradient from
// one term.  One warp per tile; the body is fsym_tile with KE.
template <int N, int MINW, bool SKET>
__global__ void __launch_bounds__(32, MINW) gsym_kernel(const int2 *__restrict__ tiles, int ntiles,
                                                   int LC, int K, int nst, Consts<N> cs,
                                                   const double *__restrict__ bra,
                                                   const double *__restrict__ ket,
                                                   const double *__restrict__ C,
                                                   const double *__restrict__ scal, RawMap kmap,
                                                   double *__restrict__ part_b,
                                                   double *__restrict__ part_k, int *status) {
    __shared__ double sacc[2 * SumFields<N>::size * 32];
    __shared__ double krow[ket_table<N>(1)];
    __shared__ double kred[ket_red<N>()];
    __shared__ __align__(16) double sket[SKET ? 2 * KetLayout<N>::size : 2];
    const int t = blockIdx.x;
    if (t >= ntiles) return;
    fsym_tile<N, true, false, SKET, true, true>(t, tiles[t], LC, K, nst, cs, bra, ket, C, kmap, nullptr, nullptr,
                                                part_b, part_k, status, FusedSmem{sacc, krow, kred, sket}, false,
                                                nullptr, 0, -1, TileOut{}, scal[0]);
}

// Fused pass over unordered pairs (k >= l): one warp per tile; the body is
// fsym_tile (necg_device.cuh), shared with the batched persistent kernel.
// blockIdx.y = pc splits the symmetry terms of every tile over npc warps (a
// small basis then still fills the GPU): split pc takes terms [pc PC, pc PC +
// PC), writes its partials to slot t npc + pc and its H, S sums to H, S + pc K^2
// (to be summed by hs_reduce_kernel); npc = 1 is the unsplit pass.
template <int N, int MINW, bool VKET, bool SKET>
__global__ void __launch_bounds__(32, MINW) fsym_kernel(const int2 *__restrict__ tiles, int t_begin, int t_end,
                                                   int LC, int K, int nst, int npc, Consts<N> cs,
                                                   const double *__restrict__ bra,
                                                   const double *__restrict__ ket,
                                                   const double *__restrict__ C, RawMap kmap,
                                                   double *__restrict__ H, double *__restrict__ S,
                                                   double *__restrict__ part_b,
                                                   double *__restrict__ part_k, int *status) {
    __shared__ double sacc[2 * SumFields<N>::size * 32];
    __shared__ double krow[ket_table<N>(2)];
    __shared__ double kred[ket_red<N>()];
    __shared__ __align__(16) double sket[SKET ? 2 * KetLayout<N>::size : 2];
    const int t = t_begin + blockIdx.x;
    if (t >= t_end) return;
    const int pc = blockIdx.y, PC = (nst + npc - 1) / npc;
    const int p0 = min(pc * PC, nst), p1 = min(p0 + PC, nst);
    const size_t off = (size_t)pc * K * K;
    fsym_tile<N, VKET, false, SKET>(t * npc + pc, tiles[t], LC, K, nst, cs, bra, ket, C, kmap, H ? H + off : nullptr,
                                    H ? S + off : nullptr, part_b, part_k, status,
                                    FusedSmem{sacc, krow, kred, sket}, false, nullptr, p0, p1);
}

// H, S = sum over the npc splits of the fused pass (fixed order: deterministic).
__global__ void __launch_bounds__(256) hs_reduce_kernel(const double *__restrict__ Hp,
                                                        const double *__restrict__ Sp, int npc, size_t KK,
                                                        double *__restrict__ H, double *__restrict__ S) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < KK; i += (size_t)gridDim.x * blockDim.x) {
        double h = Hp[i], s = Sp[i];
        for (int pc = 1; pc < npc; ++pc) {
            h += Hp[pc * KK + i];
            s += Sp[pc * KK + i];
        }
        H[i] = h;
        S[i] = s;
    }
}

// The fused pass with W-warp blocks (W = 8, 12 or 16), one per SM, persistent over
// the queue of tile groups (fsym_group).  The warps of a block meet only at the
// ends of a unit: a block barrier per term, which once kept the warps of a scheduler
// in step, now only costs (LiH K = 1024 on a B200, an earlier form of the term: 2.54
// ms with it, 2.76 ms and more with half of the warps taking it in mid-term, 2.34
// ms without).  KE: the symmetric pass with E known.
template <int N, int WARPS, bool KE = false>
__global__ void __launch_bounds__(32 * WARPS, 1) fsym_block_kernel(const int2 *__restrict__ groups, int ngroups,
                                                                int *__restrict__ qcount,
                                                                const int *__restrict__ tstart, int LC, int K,
                                                                int nst, Consts<N> cs,
                                                                const double *__restrict__ bra,
                                                                const double *__restrict__ ket,
                                                                const double *__restrict__ C, RawMap kmap,
                                                                double *__restrict__ H, double *__restrict__ S,
                                                                double *__restrict__ part_b,
                                                                double *__restrict__ part_k, int *status,
                                                                double *__restrict__ xsym, int tail0,
                                                                const double *__restrict__ scal) {
    extern __shared__ __align__(16) double smem[];
    __shared__ int gsh;
    for (;;) {
        if (threadIdx.x == 0) gsh = atomicAdd(qcount, 1);
        __syncthreads();
        const int g = gsh;
        __syncthreads();  // every thread has read gsh before it changes
        if (g >= ngroups) break;
        fsym_group<N, WARPS, KE>(g, groups[g], tail0, tstart, LC, K, nst, cs, bra, ket, C, kmap, H, S, part_b, part_k,
                                 status, xsym, KE ? scal[0] : 0.0, smem);
    }
}

// H and S of the tiles of the block variants' split tail: block = one tile (tail
// group j, warp w).
template <int N>
__global__ void __launch_bounds__(256) fsym_tail_fix_kernel(const int2 *__restrict__ groups, int tail0, int W,
                                                            int LC, int K, const double *__restrict__ xsym,
                                                            double *__restrict__ H, double *__restrict__ S) {
    const int j = blockIdx.x / W, w = blockIdx.x - j * W;
    fix_tail_tile<N>(groups[tail0 + j * sgroup_parts(groups[tail0])], j, w, W, LC, K, xsym, H, S);
}

// Partials of the fused (KE = false) or the symmetric pass into the per-basis
// sums: block (kb, f) (sum_partials).  The symmetric pass has no row field.
template <int N, bool KE>
__global__ void __launch_bounds__(256) fsym_sum_kernel(PassParts p, double *__restrict__ sums) {
    __shared__ double red[4][8][32];
    sum_partials<N, !KE>(p, blockIdx.x, blockIdx.y, sums, red);
}

// rows[i] = (H C)_i, rows[K + i] = (S C)_i from the per-basis sums (a shard's share).
template <int N>
__global__ void __launch_bounds__(128) rows_from_sums_kernel(const double *__restrict__ sums, int K,
                                                             double *__restrict__ rows) {
    constexpr int PB = SumFields<N>::size, R = SumFields<N>::row;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * K) return;
    const int which = i >= K, m = i - which * K;
    rows[i] = sums[(size_t)(which * PB + R) * K + m] + sums[(size_t)((2 + which) * PB + R) * K + m];
}

// From the per-basis sums to the gradient, 32 bases per block (finish_block).
// OWN_E: every block forms E and norm from the row sums (the same order in each,
// 5 K reads that cost less than a kernel of their own), block 0 writes them and f,
// and GRADC of the block's bases goes to gradc; else E and norm are scal's (KE:
// the sums are combined already).
template <int N, bool KE, bool OWN_E>
__global__ void __launch_bounds__(256) fsym_finish_kernel(const double *__restrict__ sums, int K, Consts<N> cs,
                                                          const double *__restrict__ bra,
                                                          const double *__restrict__ C, double *__restrict__ scal,
                                                          int folded, double *__restrict__ fields,
                                                          double *__restrict__ g, double *__restrict__ gradc,
                                                          double *__restrict__ f_out, int *status) {
    extern __shared__ __align__(16) double smem[];
    __shared__ double sh[2][32], en[4];
    if (OWN_E) {
        energy_from_rows<N>(sums, C, K, sh, en);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) scal[i] = en[i];
            if (f_out) *f_out = en[0];
            if (!isfinite(en[0])) atomicOr(status, 2);
        }
        const int k = blockIdx.x * 32 + threadIdx.x;
        if (threadIdx.x < 32 && k < K) gradc[k] = gradc_from_rows<N>(sums, K, k, en);
    }
    const double E = OWN_E ? en[0] : scal[0], norm = OWN_E ? en[1] : scal[1];
    if (!finish_block<N>(sums, K, bra, C, cs, folded, KE ? 0.0 : 2.0 * E, norm, blockIdx.x, fields, g, smem))
        atomicOr(status, 2);
}

// Sum the gradient-tile partials over the ket chunks, in place into chunk 0:
// one thread per (field, k), coalesced along k.
__global__ void __launch_bounds__(256) grad_sum_kernel(double *__restrict__ part, int nlc, int K,
                                                       int PS) {
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)PS * K) return;
    double s = part[id];
    const size_t stride = (size_t)PS * K;
    for (int lc = 1; lc < nlc; ++lc) s += part[id + lc * stride];
    part[id] = s;
}

// Scale the summed partial of basis k by norm C_k (python/make_grad.py:61-79)
// and write GRADA block k in the reference's parameter order.
template <int N>
__global__ void __launch_bounds__(128) grad_reduce_kernel(const double *__restrict__ part, int K,
                                                          const double *__restrict__ bra,
                                                          const double *__restrict__ C,
                                                          const double *__restrict__ scal,
                                                          double *__restrict__ g, int *status) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const double sc = scal[1] * (C ? C[k] : 1.0);
    if (!grad_reduce_at<N>(part, 1, K, bra_at<N>(bra, K, k), 32, sc, g, k)) atomicOr(status, 2);
}

// python/rrms.py:21-120 rrms(stfe, stf, ii, jj, n1) per term: terms[5 t ..] =
// (stfe, stf, ii, jj, n1), 1-based; out[2 t] = ov, out[2 t + 1] = st[n1] ov.
template <int N>
__global__ void __launch_bounds__(128) rrms_kernel(const int *__restrict__ terms, int nterms, int K,
                                                   int nst, Consts<N> cs,
                                                   const double *__restrict__ ket,
                                                   double *__restrict__ out, int *status) {
    using KL = KetLayout<N>;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nterms) return;
    const int *q = terms + 5 * t;
    const int stfe = q[0] - 1, stf = q[1] - 1, ii = q[2] - 1, jj = q[3] - 1, n1 = q[4] - 1;
    if (stfe < 0 || stfe >= nst || stf < 0 || stf >= nst || ii < 0 || ii >= K || jj < 0 || jj >= K ||
        n1 < 0 || n1 >= 3 * N) {
        atomicOr(status, 4);
        out[2 * t] = out[2 * t + 1] = NAN;
        return;
    }
    double T[3 * N], ov;
    const bool ok = term_dipole<N, double>(ket + ((size_t)ii * nst + stfe) * KL::size,
                                           ket + ((size_t)jj * nst + stf) * KL::size, cs, T, ov);
    double tn = T[0];
#pragma unroll
    for (int m = 1; m < 3 * N; ++m)
        if (m == n1) tn = T[m];
    out[2 * t] = ov;
    out[2 * t + 1] = tn * ov;
    if (!ok) flag_status(status, 1, ii * K + jj);
}

// Dipole sums of python/necg.py:200-244 contracted with C on the fly, over the
// energy tiles (lower triangle): for every pair k >= l and every (Pe, P),
// weight (2 - delta_kl) C_k C_l scvv[Pe] scvv[P]; den += w ov and
// num[m] += w st[m] ov.  One warp per tile; the warp's sums go to
// part[t * (3N + 1) + m] (m = 0: den) in a fixed shuffle order.
template <int N>
__global__ void __launch_bounds__(32) dipole_kernel(const int2 *__restrict__ tiles, int ntiles, int LC,
                                                    int K, int nst, Consts<N> cs,
                                                    const double *__restrict__ ket,
                                                    const double *__restrict__ C,
                                                    double *__restrict__ part, int *status) {
    using KL = KetLayout<N>;
    constexpr int NM = 3 * N + 1;
    const int t = blockIdx.x;
    const int lane = threadIdx.x;
    if (t >= ntiles) return;
    const int2 tl = tiles[t];
    int k, l0, lend;
    double acc[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[m] = 0.0;
    bool ok = true;
    if (energy_lane_range(tl.x, tl.y, lane, LC, K, k, l0, lend)) {
        const double Ck = C[k];
        for (int Pe = 0; Pe < nst; ++Pe) {
            const double *kb = ket + ((size_t)k * nst + Pe) * KL::size;
            const double wek = kb[KL::w] * Ck;
            for (int l = l0; l < lend; ++l) {
                const double wl = (l == k ? 1.0 : 2.0) * wek * C[l];
                for (int P = 0; P < nst; ++P) {
                    const double *kr = ket + ((size_t)l * nst + P) * KL::size;
                    double T[3 * N], ov;
                    ok = term_dipole<N, double>(kb, kr, cs, T, ov) && ok;
                    const double wo = wl * kr[KL::w] * ov;
                    acc[0] += wo;
#pragma unroll
                    for (int m = 0; m < 3 * N; ++m) acc[1 + m] += wo * T[m];
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < NM; ++m) {
        double v = acc[m];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) part[(size_t)t * NM + m] = v;
    }
    if (!ok) flag_status(status, 1, k * K + l0);
}

// The same sums when the symmetry set is a group whose shift maps follow its
// coordinate maps.  Then (Pe k | Q Pe l) = (k | Q l) up to Pe: B, e and T of the
// pair are those of (k, Q l) in Pe's frame, so the nst^2 terms of a pair fall into
// nst classes Q with one overlap and one T each,
//   den += c_Q ov_Q,  num += ov_Q R_Q T_Q,  c_Q = sum_Pe w_Pe w_QPe,
//   R_Q = sum_Pe w_Pe w_QPe Pe^-1
// (cls: c_Q and R_Q, N x N row-major, per class).  R_Q multiplies the sums over
// the tile's kets.  FP64-latency bound at small K, so the classes are split over
// blockIdx.y until the GPU is full; partials at slot t gridDim.y + blockIdx.y.
// LiH K = 160 on a B200: the whole call 829 -> 106 us (24 instead of 576 terms per pair).
template <int N>
__global__ void __launch_bounds__(32) dipole_group_kernel(const int2 *__restrict__ tiles, int ntiles, int LC, int K,
                                                          int nst, Consts<N> cs, const double *__restrict__ bra,
                                                          const double *__restrict__ ket,
                                                          const double *__restrict__ C,
                                                          const double *__restrict__ cls,
                                                          double *__restrict__ part, int *status) {
    using KL = KetLayout<N>;
    constexpr int NM = 3 * N + 1;
    const int t = blockIdx.x, lane = threadIdx.x;
    if (t >= ntiles) return;
    const int2 tl = tiles[t];
    const int q0 = blockIdx.y * nst / gridDim.y, q1 = (blockIdx.y + 1) * nst / gridDim.y;
    int k, l0, lend;
    double num[3 * N], den = 0.0;
#pragma unroll
    for (int m = 0; m < 3 * N; ++m) num[m] = 0.0;
    bool ok = true;
    if (energy_lane_range(tl.x, tl.y, lane, LC, K, k, l0, lend)) {
        const double Ck = C[k];
        const BraRef b{bra_at<N>(bra, K, k)};
        for (int q = q0; q < q1; ++q) {
            double a[3 * N], a0 = 0.0;
#pragma unroll
            for (int m = 0; m < 3 * N; ++m) a[m] = 0.0;
            for (int l = l0; l < lend; ++l) {
                double Bi[tri(N)], T[3 * N], ov;
                ok = term_core<N, double>(b, ket + ((size_t)l * nst + q) * KL::size, Bi, T, ov) && ok;
                const double wo = (l == k ? 1.0 : 2.0) * Ck * C[l] * ov;
                a0 += wo;
#pragma unroll
                for (int m = 0; m < 3 * N; ++m) a[m] += wo * T[m];
            }
            const double *c = cls + (size_t)q * (N * N + 1);
            den += c[0] * a0;
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const double r = c[1 + i * N + j];
#pragma unroll
                    for (int x = 0; x < 3; ++x) num[3 * i + x] += r * a[3 * j + x];
                }
        }
    }
    double *out = part + ((size_t)t * gridDim.y + blockIdx.y) * NM;
#pragma unroll
    for (int m = 0; m < NM; ++m) {
        double v = m == 0 ? den : num[m - 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) out[m] = v;
    }
    if (!ok) flag_status(status, 1, k * K + l0);
}

// Sum the dipole tile partials in a fixed order (one block) and form
// comps[m] = num[m] / den (0 when den = 0, as python/necg.py:228) and the
// dipole d_c = sum_i ncv[i + 1] comps[3 i + c].
template <int N>
__global__ void __launch_bounds__(1024) dipole_sum_kernel(const double *__restrict__ part, int nslots, Consts<N> cs,
                                                          double *__restrict__ comps, double *__restrict__ dip) {
    constexpr int NM = 3 * N + 1;
    constexpr int F = NM <= 16 ? 16 : 32, ROWS = 1024 / F;  // F fields side by side, every ROWS-th slot per thread
    __shared__ double red[ROWS][F + 1];
    __shared__ double tot[NM];
    const int m = threadIdx.x % F, r = threadIdx.x / F;
    double s = 0.0;
    if (m < NM) {
#pragma unroll 8
        for (int t = r; t < nslots; t += ROWS) s += part[(size_t)t * NM + m];
    }
    red[r][m] = s;
    __syncthreads();
    for (int w = ROWS / 2; w > 0; w >>= 1) {
        if (r < w) red[r][m] += red[r + w][m];
        __syncthreads();
    }
    const int j = threadIdx.x;
    if (j < NM) tot[j] = red[0][j];
    __syncthreads();
    if (j < 3 * N) comps[j] = tot[0] != 0.0 ? tot[1 + j] / tot[0] : 0.0;
    __syncthreads();
    if (j < 3 && dip) {
        double d = 0.0;
        for (int i = 0; i < N; ++i) d += cs.q[i] * (tot[0] != 0.0 ? tot[1 + 3 * i + j] / tot[0] : 0.0);
        dip[j] = d;
    }
}

// Per-term elements for the matel / gradel API: terms[3 t .. 3 t + 2] =
// (stf, ii, jj), 1-based as in python/matel.py:28 and python/gradel.py:27.
template <int N>
__global__ void __launch_bounds__(128) matel_kernel(const int *__restrict__ terms, int nterms, int K,
                                                    int nst, Consts<N> cs,
                                                    const double *__restrict__ bra,
                                                    const double *__restrict__ ket,
                                                    double *__restrict__ out, int *status) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nterms) return;
    const int stf = terms[3 * t] - 1, ii = terms[3 * t + 1] - 1, jj = terms[3 * t + 2] - 1;
    if (stf < 0 || stf >= nst || ii < 0 || ii >= K || jj < 0 || jj >= K) {
        atomicOr(status, 4);
        for (int q = 0; q < 4; ++q) out[4 * t + q] = NAN;
        return;
    }
    const double *kr = ket + ((size_t)jj * nst + stf) * KetLayout<N>::size;
    if (!matel_one<N, double>(BraRef{bra_at<N>(bra, K, ii)}, kr, cs, out + 4 * t))
        flag_status(status, 1, ii * K + jj);
}

template <int N>
__global__ void __launch_bounds__(128) gradel_kernel(const int *__restrict__ terms, int nterms,
                                                     int K, int nst, Consts<N> cs,
                                                     const double *__restrict__ bra,
                                                     const double *__restrict__ ket,
                                                     double *__restrict__ tgvl,
                                                     double *__restrict__ tgvls, int *status) {
    constexpr int blk = tri(N) + 3 * N;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nterms) return;
    const int stf = terms[3 * t] - 1, ii = terms[3 * t + 1] - 1, jj = terms[3 * t + 2] - 1;
    if (stf < 0 || stf >= nst || ii < 0 || ii >= K || jj < 0 || jj >= K) {
        atomicOr(status, 4);
        for (int q = 0; q < blk; ++q) tgvl[(size_t)t * blk + q] = tgvls[(size_t)t * blk + q] = NAN;
        return;
    }
    const double *kr = ket + ((size_t)jj * nst + stf) * KetLayout<N>::size;
    double L[tri(N)];
#pragma unroll
    for (int q = 0; q < tri(N); ++q) L[q] = bra_at<N>(bra, K, ii)[(BraLayout<N>::L + q) * 32];
    if (!gradel_one<N, double>(BraRef{bra_at<N>(bra, K, ii)}, kr, cs, L, ii == jj,
                               tgvl + (size_t)t * blk, tgvls + (size_t)t * blk))
        flag_status(status, 1, ii * K + jj);
}

// FP64 throughput probe: 8 independent FMA chains per thread, all in
// registers.  Used to measure the FP64 roofline denominator on the running GPU.
__global__ void __launch_bounds__(256) fp64_probe_kernel(int iters, double seed, double *sink) {
    double a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = seed + threadIdx.x * 1e-7 + j;
    const double b = 0.999999999, c = 1e-9;
    for (int i = 0; i < iters; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = fma(a[j], b, c);
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += a[j];
    if (s == 12345.6789) sink[blockIdx.x] = s;  // never true; keeps the chains live
}

// Boys function on an array (python/utils.py:78-106)
__global__ void f0_kernel(const double *__restrict__ z, int count, double *__restrict__ f,
                          double *__restrict__ df) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    double fs, D2, ia, zo;
    boys<true>(1.0, z[i], fs, D2, ia, zo);  // a = 1: fs = F0(z), D2 = 2 F0'(z) / F0(z)
    if (f) f[i] = fs;
    if (df) df[i] = 0.5 * fs * D2;
}

// ---------------------------------------------------------------------------
// Host-side launchers (one instantiation per supported particle count)
template <int N> Consts<N> make_consts(const double *mass, const double *ncv, double efs) {
    Consts<N> c;
    for (int i = 0; i < N * N; ++i) c.M[i] = mass[i];
    for (int q = 1; q <= N; ++q)
        for (int p = 0; p < q; ++p) c.cv[vidx(p, q)] = 2.0 * ncv[p] * ncv[q] / NECG_SQRT_PI;
    for (int i = 0; i < N; ++i) c.q[i] = ncv[i + 1];
    c.efs = efs;
    c.sqrt8n = sqrt(pow(8.0, N));
    return c;
}

// SMs of the current device.
int device_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

template <int N> struct Launch {
    static void prep(const LaunchArgs &a, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        const int nbb = (a.K + 63) / 64, nbk = (a.K * a.nst + 63) / 64;
        prep_kernel<N><<<nbb + nbk, 64, 0, st>>>(a.iv, a.C, a.K, a.nst, nbb, cs, a.sml, a.sms, a.scvv, a.pinv,
                                                 a.sms_general, a.bra, a.ket, a.status, a.qcount);
    }
    template <int MINW> static void energy_v(const LaunchArgs &a, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        energy_kernel<N, MINW><<<a.ntiles, 32, 0, st>>>(a.tiles, a.ntiles, a.LC_e, a.K, a.nst, cs, a.bra,
                                                        a.ket, a.H, a.S, a.Kin, a.Pot, a.status);
    }
    template <int W> static void energy_split(const LaunchArgs &a, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        energy_split_kernel<N, W><<<a.ntiles, 32 * W, 0, st>>>(a.tiles, a.LC_e, a.K, a.nst, cs, a.bra, a.ket, a.H, a.S,
                                                               a.Kin, a.Pot, a.status);
    }
    static void energy(const LaunchArgs &a, cudaStream_t st) {
        switch (energy_warps(a.nst, a.ntiles, device_sms())) {
        case 2: energy_split<2>(a, st); return;
        case 4: energy_split<4>(a, st); return;
        case 8: energy_split<8>(a, st); return;
        }
        switch (a.minb_e) {
        case 12: energy_v<12>(a, st); break;
        case 16: energy_v<16>(a, st); break;
        case 20: energy_v<20>(a, st); break;
        default: energy_v<8>(a, st); break;
        }
    }
    template <int MINW> static void grad_v(const LaunchArgs &a, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        const int nkb = (a.K + 31) / 32, nlc = (a.K + a.LC_g - 1) / a.LC_g;
        grad_kernel<N, MINW><<<nkb * nlc, 32, 0, st>>>(nkb, nlc, a.LC_g, a.K, a.nst, cs, a.bra, a.ket, a.scal, a.lam,
                                                       a.part, a.status);
    }
    // variant codes: warps per SM the kernel is compiled for (100 + w: the same
    // as w); 168 registers spill the n > 3 term (LiH K = 700, chunk 4: 2.00 ms at 8
    // warps per SM, 2.61 at 12) and 128 more so: 16 and 20 run 12 there
    static void grad_tiles(const LaunchArgs &a, cudaStream_t st) {
        const int w = a.minb_g % 100;
        if (w == 8) grad_v<8>(a, st);
        else if (w == 12 || N > 3) grad_v<12>(a, st);
        else grad_v<N <= 3 ? 16 : 12>(a, st);
    }
    static void grad_reduce(const LaunchArgs &a, cudaStream_t st) {
        const int nlc = (a.K + a.LC_g - 1) / a.LC_g;
        constexpr int PS = Part<N>::size;
        const size_t nthr = (size_t)PS * a.K;
        if (nlc > 1) grad_sum_kernel<<<(unsigned)((nthr + 255) / 256), 256, 0, st>>>(a.part, nlc, a.K, PS);
        grad_reduce_kernel<N><<<(a.K + 127) / 128, 128, 0, st>>>(a.part, a.K, a.bra, a.C, a.scal, a.g,
                                                                  a.status);
    }
    template <int MINW, bool SKET> static void gsym_v(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
            gsym_kernel<N, MINW, SKET><<<a.nstiles, 32, 0, st>>>(a.stiles, a.nstiles, a.LC_s, a.K, a.nst, cs, a.bra,
                                                                 a.ket, a.C, a.scal, a.kmap, a.psym,
                                                                 a.psym + (size_t)a.nstiles * 2 * SumFields<N>::size * 32,
                                                                 a.status);
        }
    }
    // blocks when the handle's groups are 8 chunks wide, for n > 3 (LiH K = 400, ket
    // chunk 2: 434 us for the gradient against 578 to 621 of the one-warp tiles; H2
    // K = 2048, chunk 4, measured with an earlier term: 709 against 653)
    static bool gsym_block(const LaunchArgs &a) {
        return N > 3 && a.minb_s >= 200 && fused_block_warps(a.minb_s) == 8 && a.sgroups && a.qcount && a.urange;
    }
    static void gsym_tiles(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (N > 3)
            if (gsym_block(a)) {
                fsym_block<8, true>(a, st);
                return;
            }
        // A handle tuned to a block variant at n <= 3 takes one-warp tiles with staged ket
        // records, 12 to the SM once they are more than 8 to the SM (the gradient of H2 K =
        // 2048, chunk 4: 716 us, 756 at 8 to the SM, 734 at 16; H2 K = 300, chunk 1: 63.5,
        // 67.8 and 65.5; He K = 2032, chunk 8: 250, 249 and 254), where they are fewer 8,
        // whose wider register budget has the shorter chain (H2 K = 600, chunk 8: 139 us,
        // 143 at 12; H2 K = 300, chunk 4: 76 and 82).
        if (N <= 3 && a.minb_s >= 200) {
            if (a.nstiles > 8 * device_sms()) gsym_v<12, true>(a, st);
            else gsym_v<8, true>(a, st);
            return;
        }
        switch (a.minb_s) {
        case 12:
        case 112: gsym_v<12, false>(a, st); break;
        case 16: gsym_v<16, false>(a, st); break;
        case 118: gsym_v<8, true>(a, st); break;
        case 122: gsym_v<12, true>(a, st); break;
        default: gsym_v<8, false>(a, st); break;
        }
    }
    static void gsym_reduce(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            sum<true>(a, gsym_block(a), 1, 0, a.nstiles, st);
            finish<true, false>(a, nullptr, nullptr, st);
        }
    }
    // the per-basis sums; blocks: the pass ran as a block variant over the whole tile list
    template <bool KE>
    static void sum(const LaunchArgs &a, bool blocks, int npc, int t0, int t1, cudaStream_t st) {
        constexpr int PB = SumFields<N>::size;
        const bool tail = blocks && a.sg_ntail > 0 && a.sg_parts >= 2;
        const PassParts p{a.stile_start, blocks ? a.urange : nullptr, tail ? a.tslot : nullptr, a.psym,
                          a.psym + (size_t)a.nstiles * npc * 2 * PB * 32, a.xsym, a.LC_s, a.K, t0, t1, npc, a.sg_parts};
        fsym_sum_kernel<N, KE><<<dim3((a.K + 31) / 32, KE ? PB - 1 : PB), 256, 0, st>>>(p, a.part);
    }
    template <bool KE, bool OWN_E>
    static void finish(const LaunchArgs &a, double *f_out, double *gradc, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        constexpr int smem = FinishSmem<N>::size * 8;
        fsym_finish_kernel<N, KE, OWN_E><<<(a.K + 31) / 32, 256, smem, st>>>(a.part, a.K, cs, a.bra, a.C, a.scal,
                                                                            a.kmap.fold, a.sums, a.g, gradc, f_out,
                                                                            a.status);
    }
    template <int MINW, bool VKET, bool SKET = false> static void fsym_v(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
            const int t0 = a.st_end > 0 ? a.st_begin : 0, t1 = a.st_end > 0 ? a.st_end : a.nstiles;
            if (t1 <= t0) return;
            const int npc = a.npc > 1 ? a.npc : 1;
            fsym_kernel<N, MINW, VKET, SKET><<<dim3(t1 - t0, npc), 32, 0, st>>>(
                a.stiles, t0, t1, a.LC_s, a.K, a.nst, npc, cs, a.bra, a.ket, a.C, a.kmap, npc > 1 && a.H ? a.Hp : a.H,
                npc > 1 && a.H ? a.Sp : a.S, a.psym, a.psym + (size_t)a.nstiles * npc * 2 * SumFields<N>::size * 32, a.status);
        }
    }
    template <int WARPS, bool KE = false> static void fsym_block(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            constexpr int smem = fsym_block_smem_bytes<N>(WARPS);
            if constexpr (smem <= 232448) {
                auto kern = fsym_block_kernel<N, WARPS, KE>;
                int dev = 0;
                cudaGetDevice(&dev);
                // the shared-memory opt-in is per device: once per instantiation and device
                static bool attr[64] = {};
                if (dev < 0 || dev >= 64 || !attr[dev]) {
                    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
                    if (dev >= 0 && dev < 64) attr[dev] = true;
                }
                const int sms = device_sms();
                Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
                // the fused sequence's prep has reset the queue; the gradient alone comes later
                if (KE) cudaMemsetAsync(a.qcount, 0, sizeof(int), st);
                const int grid = a.nsgroups < sms ? a.nsgroups : sms;
                if (grid < 1) return;
                kern<<<grid, 32 * WARPS, smem, st>>>(a.sgroups, a.nsgroups, a.qcount, a.stile_start, a.LC_s, a.K,
                                                     a.nst, cs, a.bra, a.ket, a.C, a.kmap, a.H, a.S, a.psym,
                                                     a.psym + (size_t)a.nstiles * 2 * SumFields<N>::size * 32, a.status,
                                                     a.xsym, a.sg_tail0, a.scal);
            }
        }
    }
    static void fsym_tiles(const LaunchArgs &a, cudaStream_t st) {
        if (a.minb_s >= 200 && a.st_end == 0 && a.sgroups && a.qcount) {
            const int w = fused_block_warps(a.minb_s);  // 2xy: block variants
            if (w == 16) fsym_block<16>(a, st);
            else if (w == 12) fsym_block<12>(a, st);
            else fsym_block<8>(a, st);
            return;
        }
        switch (a.minb_s) {  // 100 + w: ket records read at the point of use
        case 12: fsym_v<12, false>(a, st); break;
        case 16: fsym_v<16, false>(a, st); break;
        case 108: fsym_v<8, true>(a, st); break;
        case 112: fsym_v<12, true>(a, st); break;
        case 118: fsym_v<8, true, true>(a, st); break;
        case 122: fsym_v<12, true, true>(a, st); break;
        default: fsym_v<8, false>(a, st); break;
        }
    }
    static void fsym_tail(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            const int W = fused_block_warps(a.minb_s);
            fsym_tail_fix_kernel<N><<<a.sg_ntail * W, 256, 0, st>>>(a.sgroups, a.sg_tail0, W, a.LC_s, a.K, a.xsym, a.H,
                                                                    a.S);
        }
    }
    static void fsym_sum(const LaunchArgs &a, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            const int t0 = a.st_end > 0 ? a.st_begin : 0, t1 = a.st_end > 0 ? a.st_end : a.nstiles;
            const int npc = a.npc > 1 && a.minb_s < 200 ? a.npc : 1;
            const bool blocks = a.minb_s >= 200 && a.st_end == 0 && a.sgroups && a.urange;
            sum<false>(a, blocks, npc, t0, t1, st);
        }
    }
    static void fsym_finish(const LaunchArgs &a, double *f_out, double *gradc, bool own_e, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32) {
            if (own_e) finish<false, true>(a, f_out, gradc, st);
            else finish<false, false>(a, f_out, gradc, st);
        }
    }
    static void rows_from_sums(const LaunchArgs &a, double *rows, cudaStream_t st) {
        if constexpr (Part<N>::size <= 32)
            rows_from_sums_kernel<N><<<(2 * a.K + 127) / 128, 128, 0, st>>>(a.part, a.K, rows);
    }
    static void rrms(const LaunchArgs &a, const int *terms, int nterms, double *out, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        rrms_kernel<N><<<(nterms + 127) / 128, 128, 0, st>>>(terms, nterms, a.K, a.nst, cs, a.ket, out,
                                                             a.status);
    }
    static void dipole(const LaunchArgs &a, double *part, size_t cap, double *comps, double *dip, cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        int slots = a.ntiles;
        if (a.dip_cls) {
            // classes split so that there are about 16 one-warp blocks per SM (the
            // partials must fit the workspace)
            int split = (16 * device_sms() + a.ntiles - 1) / a.ntiles;
            const size_t fit = cap / ((size_t)a.ntiles * (3 * N + 1));
            if (split > a.nst) split = a.nst;
            if ((size_t)split > fit) split = (int)fit;
            if (split < 1) split = 1;
            dipole_group_kernel<N><<<dim3(a.ntiles, split), 32, 0, st>>>(a.tiles, a.ntiles, a.LC_e, a.K, a.nst, cs,
                                                                        a.bra, a.ket, a.C, a.dip_cls, part, a.status);
            slots = a.ntiles * split;
        } else {
            dipole_kernel<N><<<a.ntiles, 32, 0, st>>>(a.tiles, a.ntiles, a.LC_e, a.K, a.nst, cs, a.ket, a.C, part,
                                                      a.status);
        }
        dipole_sum_kernel<N><<<1, 1024, 0, st>>>(part, slots, cs, comps, dip);
    }
    static void reduce_sums(const LaunchArgs &a, const double *sums, cudaStream_t st) {
        grad_reduce_kernel<N><<<(a.K + 127) / 128, 128, 0, st>>>(sums, a.K, a.bra, a.C, a.scal, a.g, a.status);
    }
    static void matel(const LaunchArgs &a, const int *terms, int nterms, double *out,
                      cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        matel_kernel<N><<<(nterms + 127) / 128, 128, 0, st>>>(terms, nterms, a.K, a.nst, cs, a.bra,
                                                              a.ket, out, a.status);
    }
    static void gradel(const LaunchArgs &a, const int *terms, int nterms, double *tg, double *tgs,
                       cudaStream_t st) {
        Consts<N> cs = make_consts<N>(a.mass_h, a.ncv_h, a.efs);
        gradel_kernel<N><<<(nterms + 127) / 128, 128, 0, st>>>(terms, nterms, a.K, a.nst, cs, a.bra,
                                                               a.ket, tg, tgs, a.status);
    }
};

#define NECG_DISPATCH(n, call)      \
    switch (n) {                    \
    case 1: Launch<1>::call; break; \
    case 2: Launch<2>::call; break; \
    case 3: Launch<3>::call; break; \
    case 4: Launch<4>::call; break; \
    case 5: Launch<5>::call; break; \
    case 6: Launch<6>::call; break; \
    default: return -1;             \
    }

void launch_tile_list(int2 *tiles, int K, int LC, cudaStream_t st) {
    tile_list_kernel<<<row_blocks(K), 128, 0, st>>>(tiles, K, LC);
}
void launch_sym_lists(const SymQueue &q, const SymLists &o, cudaStream_t st) {
    sym_lists_kernel<<<row_blocks(q.K), 128, 0, st>>>(q, o);
}
int launch_prep(const LaunchArgs &a, cudaStream_t st) {
    NECG_DISPATCH(a.n, prep(a, st));
    return 0;
}
int launch_energy(const LaunchArgs &a, cudaStream_t st) {
    NECG_DISPATCH(a.n, energy(a, st));
    return 0;
}
int launch_grad_tiles(const LaunchArgs &a, cudaStream_t st) {
    NECG_DISPATCH(a.n, grad_tiles(a, st));
    return 0;
}
int launch_grad_reduce(const LaunchArgs &a, cudaStream_t st) {
    NECG_DISPATCH(a.n, grad_reduce(a, st));
    return 0;
}
int launch_grad(const LaunchArgs &a, cudaStream_t st) {
    if (launch_grad_tiles(a, st)) return -1;
    return launch_grad_reduce(a, st);
}
int launch_gsym(const LaunchArgs &a, cudaStream_t st) {
    if (a.n > 5 || !a.psym || !a.stiles) return -1;
    NECG_DISPATCH(a.n, gsym_tiles(a, st));
    return 0;
}
int launch_gsym_reduce(const LaunchArgs &a, cudaStream_t st) {
    if (a.n > 5) return -1;
    NECG_DISPATCH(a.n, gsym_reduce(a, st));
    return 0;
}
int fused_block_warps(int variant) { return variant == 216 ? 16 : variant == 222 || variant == 232 ? 12 : 8; }
bool fused_variant_ok(int n, int variant) {
    if (variant < 200) return true;
    if (n < 1 || n > 5) return false;
    const int warps = fused_block_warps(variant);
    int bytes = 0;
    switch (n) {
    case 1: bytes = fsym_block_smem_bytes<1>(warps); break;
    case 2: bytes = fsym_block_smem_bytes<2>(warps); break;
    case 3: bytes = fsym_block_smem_bytes<3>(warps); break;
    case 4: bytes = fsym_block_smem_bytes<4>(warps); break;
    default: bytes = fsym_block_smem_bytes<5>(warps); break;
    }
    return bytes <= 232448;
}
int launch_fsym(const LaunchArgs &a, cudaStream_t st) {
    if (a.n > 5) return -1;
    // every buffer the pass writes must be set (no launch on a null pointer); H
    // and S are written when both are
    if (!a.H != !a.S || !a.psym || !a.stiles || !a.bra || !a.ket || !a.C || !a.status) return -1;
    if (a.npc > 1 && a.minb_s < 200 && a.H && (!a.Hp || !a.Sp)) return -1;
    NECG_DISPATCH(a.n, fsym_tiles(a, st));
    return 0;
}
int launch_fsym_tail(const LaunchArgs &a, cudaStream_t st) {
    // only a block variant over the whole tile list splits its tail; the sums read
    // the parts themselves, so this is for H and S alone
    if (!a.H || a.minb_s < 200 || a.st_end > 0 || a.sg_ntail <= 0 || a.sg_parts < 2) return 0;
    if (a.n > 5 || !a.sgroups || !a.xsym || !a.S) return -1;
    NECG_DISPATCH(a.n, fsym_tail(a, st));
    return 0;
}
int launch_fsym_sum(const LaunchArgs &a, cudaStream_t st) {
    if (a.n > 5 || !a.stile_start || !a.psym || !a.part) return -1;
    NECG_DISPATCH(a.n, fsym_sum(a, st));
    return 0;
}
int launch_fsym_finish(const LaunchArgs &a, double *f_out, double *gradc, bool own_e, cudaStream_t st) {
    if (a.n > 5 || !a.part || !a.bra || !a.C || !a.scal || !a.status || (!a.sums && !a.g) || (own_e && !gradc)) return -1;
    NECG_DISPATCH(a.n, fsym_finish(a, f_out, gradc, own_e, st));
    return 0;
}
int launch_rows_from_sums(const LaunchArgs &a, double *rows, cudaStream_t st) {
    if (a.n > 5 || !a.part || !rows) return -1;
    NECG_DISPATCH(a.n, rows_from_sums(a, rows, st));
    return 0;
}
int launch_hs_reduce(const LaunchArgs &a, cudaStream_t st) {
    if (a.npc <= 1 || !a.H) return 0;  // H and S not wanted: nothing to sum
    if (!a.Hp || !a.Sp || !a.S) return -1;
    const size_t KK = (size_t)a.K * a.K;
    const size_t blocks = (KK + 255) / 256 < 4096 ? (KK + 255) / 256 : 4096;
    hs_reduce_kernel<<<(int)blocks, 256, 0, st>>>(a.Hp, a.Sp, a.npc, KK, a.H, a.S);
    return 0;
}
int launch_reduce_sums(const LaunchArgs &a, const double *sums, cudaStream_t st) {
    if (!sums || !a.bra || !a.C || !a.scal || !a.g || !a.status) return -1;
    NECG_DISPATCH(a.n, reduce_sums(a, sums, st));
    return 0;
}
int launch_rrms(const LaunchArgs &a, const int *terms, int nterms, double *out, cudaStream_t st) {
    NECG_DISPATCH(a.n, rrms(a, terms, nterms, out, st));
    return 0;
}
int launch_dipole(const LaunchArgs &a, double *part, size_t cap, double *comps, double *dip, cudaStream_t st) {
    NECG_DISPATCH(a.n, dipole(a, part, cap, comps, dip, st));
    return 0;
}
int launch_matel(const LaunchArgs &a, const int *terms, int nterms, double *out, cudaStream_t st) {
    NECG_DISPATCH(a.n, matel(a, terms, nterms, out, st));
    return 0;
}
int launch_gradel(const LaunchArgs &a, const int *terms, int nterms, double *tg, double *tgs,
                  cudaStream_t st) {
    NECG_DISPATCH(a.n, gradel(a, terms, nterms, tg, tgs, st));
    return 0;
}
void launch_rows_finalize(const LaunchArgs &a, double *f_out, double *gradc, int given, double eng,
                          double norm, cudaStream_t st, const double *given_dev, double *en_out) {
    rows_kernel<<<(a.K * 32 + 255) / 256, 256, 0, st>>>(a.H, a.S, a.C, a.K, a.rows);
    finalize_kernel<<<1, 1024, 0, st>>>(a.rows, a.C, a.K, a.scal, f_out, gradc, a.status, given, eng,
                                        norm, given_dev, en_out);
}
void launch_finalize(const LaunchArgs &a, const double *rows, double *f_out, double *gradc, cudaStream_t st) {
    finalize_kernel<<<1, 1024, 0, st>>>(rows, a.C, a.K, a.scal, f_out, gradc, a.status, 0, 0.0, 0.0, nullptr,
                                        nullptr);
}
void launch_fp64_probe(int blocks, int iters, double *sink, cudaStream_t st) {
    fp64_probe_kernel<<<blocks, 256, 0, st>>>(iters, 1.0, sink);
}
void launch_f0(const double *z, int count, double *f, double *df, cudaStream_t st) {
    f0_kernel<<<(count + 255) / 256, 256, 0, st>>>(z, count, f, df);
}

int ket_record_size(int n) {
    switch (n) {
    case 1: return KetLayout<1>::size;
    case 2: return KetLayout<2>::size;
    case 3: return KetLayout<3>::size;
    case 4: return KetLayout<4>::size;
    case 5: return KetLayout<5>::size;
    case 6: return KetLayout<6>::size;
    default: return 0;
    }
}
int bra_record_size(int n) {
    switch (n) {
    case 1: return BraLayout<1>::size;
    case 2: return BraLayout<2>::size;
    case 3: return BraLayout<3>::size;
    case 4: return BraLayout<4>::size;
    case 5: return BraLayout<5>::size;
    case 6: return BraLayout<6>::size;
    default: return 0;
    }
}
int part_stride(int n) { return n >= 1 && n <= 6 ? tri(n) + 1 + 3 * n : 0; }
size_t sums_doubles(int n, int K) { return (size_t)kSumSets * (part_stride(n) + 1) * K; }
size_t part_doubles(int n, int K) {
    const size_t ordered = (size_t)part_stride(n) * K * ((K + 3) / 4);
    const size_t sums = sums_doubles(n, K);
    return ordered > sums ? ordered : sums;
}
int ket_slots(int n) {
    switch (n) {
    case 1: return KetSlots<1>::SL;
    case 2: return KetSlots<2>::SL;
    case 3: return KetSlots<3>::SL;
    case 4: return KetSlots<4>::SL;
    default: return KetSlots<5>::SL;
    }
}
int ket_slot(int n, int f) {
    switch (n) {
    case 1: return KetSlots<1>::slot(f);
    case 2: return KetSlots<2>::slot(f);
    case 3: return KetSlots<3>::slot(f);
    case 4: return KetSlots<4>::slot(f);
    default: return KetSlots<5>::slot(f);
    }
}

}  // namespace necg
