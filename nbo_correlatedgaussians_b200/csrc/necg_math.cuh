// necg_math.cuh -- per-term FP64 math of the ECG energy+gradient path.
//
// One "term" is a (bra k, ket l, symmetry P) triple: the reference's
// matel(stf, k, l) (python/matel.py:28-210) and the bra part of
// gradel(stf, k, l) (python/gradel.py:27-392).  The reference expands every
// n x n matrix to 3n x 3n with kron(., I3) and inverts with LAPACK; here all
// work stays in n-space with the shifts viewed as n x 3 matrices, B = A_k + A_l'
// is inverted in registers (symmetric elimination), and the gradient is formed
// with respect to A_k = L_k L_k^T (a symmetric n x n matrix) and s_k, then mapped
// to vech(L_k) once per basis function (dF/dL = 2 G L).
//
// Notation (n = N particles):
//   A_k, A_l' = P^T A_l P    symmetric, packed lower (N(N+1)/2)
//   S_k, S_l' = sms s_l      n x 3 (row = particle, column = x, y, z)
//   B = A_k + A_l', Bi = B^-1, e = A_k S_k + A_l' S_l', T = Bi e   (st in the reference)
//   D_k = T - S_k, D_l = T - S_l', N = A_k M A_k, U_s = 1.5 Bi + D_s D_s^T
//   ov  = sqrt(8^n) (|L_k| |L_l|)^{3/2} / |B|^{3/2} exp(<e,T> - i1 - i2)
//   tau = 3 tr(M A_k) - 3 <N, Bi> - 2 <D_k, N D_k>,   tk = 2 ov tau
//   rho = sum_v c_v F0(|v^T T|^2 / v^T Bi v) (v^T Bi v)^{-1/2}, ert = ov rho
//   sig = efs sum_i q_i T[i,z],  zht = ov sig
//   eta = 2 tau + rho - sig,  h = tk + ert - zht = ov eta
// Coulomb pairs v: e_q (nucleus-particle) or e_p - e_q (particle-particle),
// c_v = 2 q_p q_q / sqrt(pi).
//
// Gradient.  h and ov depend on the pair through B and e alone, apart from
// factors of one side only: |L_k|^{3/2} exp(-i1) of each side, and tau, which is
// written with the bra's A_k and s_k.  With F0's derivative pieces
//   Z' = sum_v alpha_v v b_v^T - (efs/2) q e_z^T,  W = sum_v beta_v v v^T,
//   alpha_v = c_v F0'(z) a^{-3/2},  beta_v = c_v a^{-3/2} (z F0'(z) + F0(z)/2),
//   Q = Bi (Z' - 4 N D_k)
// the derivatives with respect to A_s and e_s = A_s S_s of side s = k, l through B
// and e, with the origin moved to that side's S_s, are
//   dh:  ov (Bi (6 N + W) Bi - Q D_s^T - D_s Q^T - eta U_s),  2 ov (Q + eta D_s)
//   dS: -ov U_s,                                               2 ov D_s
// (term_raw).  A basis function sums them over its terms as they are; what depends
// on its own A (the chain from e = A s, and the bra's explicit share of tau)
// multiplies only those sums, once per basis function (fold_raw, explicit_tau).
// That takes the products with A_k and A_l' and the second sandwich out of the term:
// 3238 instead of 4374 FLOP at n = 5 and 1266 instead of 1626 at n = 3.  The FP64 pipe
// bounds the pair passes; whole evaluations on a B200 went from 3.53 to 2.49 ms (LiH K
// = 1024), 1.06 to 0.72 ms (H2 K = 2048) and 0.34 to 0.22 ms (He K = 2032), the
// launches around the passes included.
// The origin: with T in the place of D_s both sides would share all values, some 400
// FLOP less at n = 5 (2.29 ms), but the sums of a function away from the origin would
// hold differences |s|^2 A times as large as themselves (components of dF/dL of tight
// functions lost 10 to 50 times the rounding error).
// The A^-1 term (coefficient D = 0.75 F) maps to vech(dF/dL) as 2 D / L_ii
// on the diagonal only, so it is kept as one scalar per basis function.
//
// All term functions are templates over the scalar type R and over the bra and
// ket accessors.  The kernels instantiate them with R = double; the operation
// counter in the C-ABI layer instantiates them with a counting scalar on the
// host, so the algorithmic FLOP count is taken from this very code.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifdef __CUDACC__
#define NECG_HD __host__ __device__ __forceinline__
#else
#define NECG_HD inline
#endif

namespace necg {

__host__ __device__ constexpr int tri(int n) { return n * (n + 1) / 2; }
// packed lower-triangular, row-major: (i, j) with i >= j
__host__ __device__ constexpr int sx(int i, int j) {
    return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

// Pade coefficients of the Boys function F0 (python/shared.py:76-86,
// source/error_function_approximation.f90) and its branch point
// (python/utils.py:85).
#define NECG_PC1 0.564691197e-04
#define NECG_PC2 0.758433197e-03
#define NECG_PC3 0.769838037e-02
#define NECG_PC4 0.629344460e-01
#define NECG_PC5 0.213271302e+00
#define NECG_PC6 0.720266520e-04
#define NECG_PC7 0.955528842e-03
#define NECG_PC8 0.101431553e-01
#define NECG_PC9 0.738522953e-01
#define NECG_PC10 0.338450368e+00
#define NECG_PC11 0.879937801e+00
#define NECG_F0_SPLIT 16.3578
#define NECG_PI 3.141592653589793
#define NECG_SQRT_PI 1.7724538509055159

// Ket record: one per (l, P), read warp-uniformly by the tile kernels (staged in
// shared memory by the block variants).  Np8 = -8 A_l' M A_l', tMA = tr(M A_l') and Sp
// are for the terms that write the kinetic part with the ket (term_value).
template <int N> struct KetLayout {
    static constexpr int T = tri(N);
    static constexpr int Ap = 0;
    static constexpr int ASp = Ap + T;
    static constexpr int i2 = ASp + 3 * N;
    static constexpr int pre = i2 + 1;
    static constexpr int w = pre + 1;    // symmetry weight scvv[P]
    static constexpr int wC = w + 1;     // 2 scvv[P] C_l (gradient weight)
    static constexpr int winv = wC + 1;  // scvv[P^-1] (ket weight of the symmetric pass)
    static constexpr int tMA = winv + 1;
    static constexpr int Np8 = tMA + 1;
    static constexpr int Sp = Np8 + T;
    static constexpr int size = (Sp + 3 * N + 1) & ~1;  // even, 16-byte records
};

// Bra record: structure of arrays by row block, field f of lane j of block kb at
// (kb size + f) 32 + j (bra_at): a warp's lanes read 256 contiguous bytes, and the
// fields of a lane are a constant distance apart, so a load needs no address
// arithmetic of its own (with a stride of K doubles the n = 3 term spent about 60
// of its 1480 instructions on addresses).
template <int N> struct BraLayout {
    static constexpr int T = tri(N);
    static constexpr int A = 0;
    static constexpr int S = A + T;
    static constexpr int AS = S + 3 * N;
    static constexpr int N8 = AS + 3 * N;  // -8 A_k M A_k
    static constexpr int i1 = N8 + T;
    static constexpr int pre = i1 + 1;     // sqrt(8^n) |L_k|^{3/2}
    static constexpr int tMA = pre + 1;
    static constexpr int term = tMA + 1;   // the fields above are all a term reads
    static constexpr int L = tMA + 1;      // L_k, packed lower
    static constexpr int size = L + T;
};

// Rows come in blocks of 32, one per lane: lane j of row block kb is basis
// 32 kb + j - row_pad(K), so that a K that is not a multiple of 32 leaves its empty
// lanes in the first block, whose rows meet the fewest kets.  (In the last block
// they would sit through all K: at K = 101 the blocks' kets add up to 212 instead
// of 293, and the pair passes take that much less.)
__host__ __device__ constexpr int row_pad(int K) { return (32 - (K & 31)) & 31; }
__host__ __device__ constexpr int row_blocks(int K) { return (K + 31) >> 5; }
// last basis of row block kb
__host__ __device__ constexpr int row_last(int K, int kb) { return 32 * kb + 31 - row_pad(K); }

// Field 0 of basis k in the blocked layout; further fields are 32 doubles apart.
template <int N, typename P> __host__ __device__ __forceinline__ P *bra_at(P *bra, int K, int k) {
    const int p = k + row_pad(K);
    return bra + (size_t)(p >> 5) * (BraLayout<N>::size * 32) + (p & 31);
}

// Per-problem constants, passed to kernels by value (constant bank).
template <int N> struct Consts {
    double M[N * N];    // inverse-mass tensor, row-major
    double cv[tri(N)];  // c_v for the n(n+1)/2 Coulomb pairs (p<q, q-major order)
    double q[N];        // ncv[1..n]
    double efs;
    double sqrt8n;      // sqrt(8^n)
};

// Doubles of one part's compact output for one tile of a split group of the
// block variants (pb fields, lc kets per tile): ket partials, then H and S sums.
__host__ __device__ inline size_t fsym_tail_slot(int pb, int lc) {
    return (size_t)lc * 2 * pb + (size_t)lc * 64;
}

// Coulomb pair enumeration order: for q = 1..N, p = 0..q-1  -> index q(q-1)/2 + p
__host__ __device__ constexpr int vidx(int p, int q) { return q * (q - 1) / 2 + p; }

// ---------------------------------------------------------------------------
// Accessors.  Bra fields are per-lane and invariant over a tile's ket loops; holding
// them in registers would cost 2 (6N + 2 tri(N)) registers, so they are re-read from
// the (L1-resident) structure-of-arrays at the point of use.  The volatile asm keeps
// the compiler from hoisting the loads out of the ket loops.  (Compiled for the host
// by the emulation of the kernels, these are plain loads.)
__device__ __forceinline__ double ldv(const double *p) {
#ifdef __CUDACC__
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
#else
    return *p;
#endif
}
// The same from shared memory.
__device__ __forceinline__ double lds(const double *p) {
#ifdef __CUDACC__
    double v;
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
#else
    return *p;
#endif
}
struct BraRef {
    const double *p;  // bra_at(bra, k)
    __device__ __forceinline__ double operator()(int f) const { return ldv(p + f * 32); }
};
// Bra record staged in shared memory (field f of this lane at p[f * 32]).
struct BraSmem {
    const double *p;  // shared base + lane
    __device__ __forceinline__ double operator()(int f) const { return lds(p + f * 32); }
};
// Ket record staged in shared memory by its warp (a broadcast load).
struct KetSmem {
    const double *p;
    __device__ __forceinline__ double operator[](int i) const { return lds(p + i); }
};
// Ket record read at the point of use (warp-uniform, L1 broadcast), so its
// fields do not stay live in registers between their uses within a term.
struct KetRefV {
    const double *p;
    __device__ __forceinline__ double operator[](int i) const { return ldv(p + i); }
};

// ---------------------------------------------------------------------------
// x^(-1/2) for normal, positive x.  On the device the hardware approximation
// rsqrt.approx.ftz.f64 (relative error below 1e-6) is refined by one step of
// Householder's third-order iteration for 1/sqrt(x): with r = 1 - x y^2,
// y <- y + y r (1/2 + 3/8 r), the series of (1 - r)^(-1/2) to second order,
// whose truncation error (of order r^3) lies far below the result's rounding.
// Measured on a B200 over 2^24 inputs in [2^-40, 2^40]: within 2 ulp of
// rsqrt(double) and 2.4 ulp of 1 / sqrt(x), at 1.56x its throughput.  Host
// builds (the emulator) use 1 / sqrt(x).
NECG_HD double rsq(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double r = fma(-(x * y), y, 1.0);
    return fma(y * r, fma(0.375, r, 0.5), y);
#else
    return 1.0 / ::sqrt(x);
#endif
}

// 1/x for normal, positive x.  On the device the hardware approximation
// rcp.approx.ftz.f64 is refined by one third-order step: with e = 1 - x y,
// y <- y + y (e + e^2), the series of 1 / (1 - e) to second order, whose
// truncation error (of order e^3) lies far below the result's rounding.  Host
// builds (the emulator) use 1 / x.
NECG_HD double rcp(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / x;
#endif
}

// Inverse Bi (packed) of a packed SPD matrix B by symmetric Gauss-Jordan
// elimination: step k takes d = B_kk, t_i = B_ik / d, B_ij -= t_i B_jk, B_ik = t_i,
// B_kk = -1 / d, and leaves -B^-1 after all of them.  The pivots d are those of
// the LDL^T factorisation (all positive iff B is positive definite; det = prod d).
// 70 products and 5 reciprocals at n = 5, against 95 and 5 inverse roots for
// Cholesky and two triangular products; its errors measured the same or smaller.
// det_m32 = det^{-3/2}.  Fully unrolled into registers.
#pragma nv_exec_check_disable
template <int N, typename R>
NECG_HD bool spd_inverse(const R (&B)[tri(N)], R (&Bi)[tri(N)], R &det_m32) {
    R a[tri(N)];
#pragma unroll
    for (int t = 0; t < tri(N); ++t) a[t] = B[t];
    bool ok = true;
    R det = R(1.0);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        R d = a[sx(k, k)];
        const bool pos = d > 0.0;
        ok = ok && pos;
        if (!pos) d = R(1.0);
        det = (k == 0) ? d : det * d;
        const R r = rcp(d);
        R t[N];
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i != k) t[i] = a[sx(i, k)] * r;
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j)
                if (i != k && j != k) a[sx(i, j)] -= t[i] * a[sx(j, k)];
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i != k) a[sx(i, k)] = t[i];
        a[sx(k, k)] = -r;
    }
#pragma unroll
    for (int t = 0; t < tri(N); ++t) Bi[t] = -a[t];
    const R y = rsq(det);
    det_m32 = (y * y) * y;
    return ok;
}

// y = S x for S symmetric (packed, read through an accessor) and x n x 3
#pragma nv_exec_check_disable
template <int N, typename R, typename Acc>
NECG_HD void symv3(const Acc &S, int off, const R (&x)[3 * N], R (&y)[3 * N]) {
    // each element of S is read once and used for the three columns (the
    // accessors may load from memory at every call)
#pragma unroll
    for (int i = 0; i < N; ++i) {
        {
            const R a = S[off + sx(i, 0)];
#pragma unroll
            for (int c = 0; c < 3; ++c) y[3 * i + c] = a * x[c];
        }
#pragma unroll
        for (int k = 1; k < N; ++k) {
            const R a = S[off + sx(i, k)];
#pragma unroll
            for (int c = 0; c < 3; ++c) y[3 * i + c] += a * x[3 * k + c];
        }
    }
}

// Boys-function pieces for one Coulomb pair.  Given a = v^T Bi v and
// bb = |v^T T|^2 (z = bb / a) returns fs = F0(z) a^{-1/2} and, when GRAD,
// D2 = 2 F0'(z) / F0(z) (so 2 F0'(z) a^{-1/2} = fs D2) and ia = 1/a.  The Pade branch
// (z <= 16.3578) and the asymptotic branch sqrt(pi/(4z)) follow
// python/utils.py:78-106; in the Pade branch F0 = sqrt(num / den), and from
// F0^2 = num / den, F0' = F0 (num'/num - den'/den) / 2, so
//   D2 = 2 F0' / F0 = (num' den - den' num) / (num den)  (Pade),  -1 / z  (asymptotic),
// with num' den - den' num evaluated as one polynomial.  Two
// special functions give every quotient and root; RCP chooses between two ways:
//   RCP:   ia = 1/a (rcp);  q = (num den a)^{-1/2} (Pade) or bb^{-1/2}:
//          fs = num q or (sqrt(pi) / 2) q, and q^2 a = 1 / (num den) or 1 / z;
//   !RCP:  ra = a^{-1/2}, ia = ra^2;  q = (num den)^{-1/2} or bb^{-1/2}:
//          fs = num q ra or (sqrt(pi) / 2) q, and q^2 = 1 / (num den) or 1 / bb.
// RCP takes four FP64 operations fewer per pair but holds more values at once;
// it is used where it timed faster on a B200 (n > 3).  The branch is taken per
// lane: every lane evaluates the Pade polynomials and the two forms differ only
// in the operand of the square root and in the factors selected, so that the
// lanes of a warp on either side of the split run the same instructions.
template <typename R> NECG_HD void boys_pade(R z, R &num, R &den) {
    num = ((((NECG_PC1 * z + NECG_PC2) * z + NECG_PC3) * z + NECG_PC4) * z + NECG_PC5) * z + 1.0;
    den = (((((NECG_PC6 * z + NECG_PC7) * z + NECG_PC8) * z + NECG_PC9) * z + NECG_PC10) * z + NECG_PC11) * z + 1.0;
}
// num' den - den' num as one polynomial of degree 10, its coefficients formed
// from the Pade coefficients when the code is compiled
struct BoysDP {
    double c[11];
    constexpr BoysDP() : c{} {
        const double nd[5] = {NECG_PC5, 2.0 * NECG_PC4, 3.0 * NECG_PC3, 4.0 * NECG_PC2, 5.0 * NECG_PC1};  // num'
        const double de[7] = {1.0, NECG_PC11, NECG_PC10, NECG_PC9, NECG_PC8, NECG_PC7, NECG_PC6};       // den
        const double dd[6] = {NECG_PC11, 2.0 * NECG_PC10, 3.0 * NECG_PC9, 4.0 * NECG_PC8, 5.0 * NECG_PC7,
                              6.0 * NECG_PC6};                                                         // den'
        const double nu[6] = {1.0, NECG_PC5, NECG_PC4, NECG_PC3, NECG_PC2, NECG_PC1};                  // num
        for (int i = 0; i < 5; ++i)
            for (int j = 0; j < 7; ++j) c[i + j] += nd[i] * de[j];
        for (int i = 0; i < 6; ++i)
            for (int j = 0; j < 6; ++j) c[i + j] -= dd[i] * nu[j];
    }
};
template <typename R> NECG_HD R boys_pade_dp(R z) {
    constexpr BoysDP p{};
    R v = R(p.c[10]) * z + p.c[9];
#pragma unroll
    for (int k = 8; k >= 0; --k) v = v * z + p.c[k];
    return v;
}
#pragma nv_exec_check_disable
template <bool GRAD, bool RCP = true, typename R>
NECG_HD void boys(R a, R bb, R &fs, R &D2, R &ia, R &z) {
    R ra = R(1.0);
    if constexpr (RCP) {
        ia = rcp(a);
    } else {
        ra = rsq(a);
        ia = ra * ra;
    }
    z = bb * ia;
    const bool pade = z <= NECG_F0_SPLIT;
    R num, den;
    boys_pade(z, num, den);
    const R c = R(0.5 * NECG_SQRT_PI);
    R q;
    if constexpr (RCP) {
        q = rsq(pade ? (num * den) * a : bb);
        fs = (pade ? num : c) * q;
    } else {
        q = rsq(pade ? num * den : bb);
        const R fp = (num * q) * ra, fa = c * q;
        fs = pade ? fp : fa;
    }
    if (GRAD) {
        const R P = boys_pade_dp(z);
        R dp, da;
        if constexpr (RCP) {
            const R qa = (q * q) * a;
            dp = qa * P;
            da = -qa;
        } else {
            const R qq = q * q;
            dp = qq * P;
            da = -(a * qq);
        }
        D2 = pade ? dp : da;
    } else {
        D2 = R(0.0);
    }
}

// Coulomb sum with the pieces of its derivative (python/gradel.py:266-337):
// returns rho = sum_v c_v F0(z_v) a_v^-1/2 and adds 2 sum_v alpha_v v b_v^T to Z
// and 2 sum_v beta_v v v^T to W (packed).
#pragma nv_exec_check_disable
template <int N, typename R>
NECG_HD R coulomb_grad(const R (&Bi)[tri(N)], const R (&T)[3 * N], const Consts<N> &cs, R (&Z)[3 * N],
                       R (&W)[tri(N)]) {
    R rho = R(0.0);
#pragma unroll
    for (int q = 1; q <= N; ++q)
#pragma unroll
        for (int p = 0; p < q; ++p) {
            R a = Bi[sx(q - 1, q - 1)];
            R bv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) bv[c] = T[3 * (q - 1) + c];
            if (p > 0) {
                a += Bi[sx(p - 1, p - 1)] - 2.0 * Bi[sx(q - 1, p - 1)];
#pragma unroll
                for (int c = 0; c < 3; ++c) bv[c] -= T[3 * (p - 1) + c];
            }
            const R bb = bv[0] * bv[0] + bv[1] * bv[1] + bv[2] * bv[2];
            R fs, D2, ia, z;
            boys<true, (N > 3)>(a, bb, fs, D2, ia, z);
            // 2 alpha = 2 c F0' a^{-3/2} = c fs D2 / a,
            // 2 beta = 2 c a^{-3/2} (z F0' + F0 / 2) = (c fs / a)(z D2 + 1)
            const R cf = cs.cv[vidx(p, q)] * fs;
            rho += cf;
            const R cfi = cf * ia;
            const R al = cfi * D2;
            const R be = al * z + cfi;
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) Z[3 * (q - 1) + cc] += al * bv[cc];
            W[sx(q - 1, q - 1)] += be;
            if (p > 0) {
#pragma unroll
                for (int cc = 0; cc < 3; ++cc) Z[3 * (p - 1) + cc] -= al * bv[cc];
                W[sx(p - 1, p - 1)] += be;
                W[sx(q - 1, p - 1)] -= be;
            }
        }
    return rho;
}

// B = A_k + A_l', its inverse, T = Bi (A_k S_k + A_l' S_l') and the overlap.
#pragma nv_exec_check_disable
template <int N, typename R, typename BA, typename KA>
NECG_HD bool term_core(const BA &b, const KA &kr, R (&Bi)[tri(N)], R (&T)[3 * N], R &ov) {
    using KL = KetLayout<N>;
    using BL = BraLayout<N>;
    R m32;
    bool ok;
    {
        R B[tri(N)];
#pragma unroll
        for (int t = 0; t < tri(N); ++t) B[t] = b(BL::A + t) + kr[KL::Ap + t];
        ok = spd_inverse<N>(B, Bi, m32);
    }
    R Ev[3 * N];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) Ev[t] = b(BL::AS + t) + kr[KL::ASp + t];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R s = Bi[sx(i, 0)] * Ev[c];
#pragma unroll
            for (int k = 1; k < N; ++k) s += Bi[sx(i, k)] * Ev[3 * k + c];
            T[3 * i + c] = s;
        }
    R i3 = Ev[0] * T[0];
#pragma unroll
    for (int t = 1; t < 3 * N; ++t) i3 += Ev[t] * T[t];
    ov = b(BL::pre) * kr[KL::pre] * m32 * exp(i3 - b(BL::i1) - kr[KL::i2]);
    return ok;
}

#pragma nv_exec_check_disable
template <int N, typename R>
NECG_HD R term_sig(const Consts<N> &cs, const R (&T)[3 * N]) {
    R sg = cs.q[0] * T[2];
#pragma unroll
    for (int i = 1; i < N; ++i) sg += cs.q[i] * T[3 * i + 2];
    return cs.efs * sg;
}

// Coulomb sum (python/matel.py:162-197)
#pragma nv_exec_check_disable
template <int N, typename R>
NECG_HD R coulomb_sum(const R (&Bi)[tri(N)], const R (&T)[3 * N], const Consts<N> &cs) {
    R r = R(0.0);
#pragma unroll
    for (int q = 1; q <= N; ++q)
#pragma unroll
        for (int p = 0; p < q; ++p) {
            R a = Bi[sx(q - 1, q - 1)];
            R bv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) bv[c] = T[3 * (q - 1) + c];
            if (p > 0) {
                a += Bi[sx(p - 1, p - 1)] - 2.0 * Bi[sx(q - 1, p - 1)];
#pragma unroll
                for (int c = 0; c < 3; ++c) bv[c] -= T[3 * (p - 1) + c];
            }
            const R bb = bv[0] * bv[0] + bv[1] * bv[1] + bv[2] * bv[2];
            R fs, D, ia, z;
            boys<false, (N > 3)>(a, bb, fs, D, ia, z);
            r += cs.cv[vidx(p, q)] * fs;
        }
    return r;
}

// 2 tau of one term, tau = 3 tr(M X) - 2 <A_s D_s, M
// A_s D_s> with X = A_k Bi A_l' = A_s - A_s Bi A_s, of either side s (D_s = T - S_s, and
// A_k D_k = -A_l' D_l).  Both subtractions cancel for the tighter side (X and T - S
// are small there against A and S, by the ratio of the exponents), so each lane
// takes the side with the smaller tr(M A): 4 tau = 12 tr(M A_s) + <-8 N_s, 1.5 Bi +
// D_s D_s^T>.  Both sides' N and S are read and one is selected (no divergent branch,
// no FP64 operation more than with a fixed side).
#pragma nv_exec_check_disable
template <int N, typename R, typename BA, typename KA>
NECG_HD R term_tau2(const BA &b, const KA &kr, const R (&Bi)[tri(N)], const R (&T)[3 * N]) {
    using BL = BraLayout<N>;
    using KL = KetLayout<N>;
    const R tl = kr[KL::tMA], tk = b(BL::tMA);
    const bool use_l = tl <= tk;
    R D[3 * N], dg = R(0.0), od = R(0.0);
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) {
        const R sl = kr[KL::Sp + t], sk = b(BL::S + t);
        D[t] = T[t] - (use_l ? sl : sk);
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            R u = 1.5 * Bi[sx(i, j)];
#pragma unroll
            for (int c = 0; c < 3; ++c) u += D[3 * i + c] * D[3 * j + c];
            const R nl = kr[KL::Np8 + sx(i, j)], nk = b(BL::N8 + sx(i, j));
            const R a = use_l ? nl : nk;
            if (i == j)
                dg = (i == 0) ? a * u : dg + a * u;
            else
                od = (i == 1) ? a * u : od + a * u;
        }
    return 6.0 * (use_l ? tl : tk) + (0.5 * dg + od);
}

// The value of one term: ov, 2 tau, rho and sig; false if B is not positive definite.
#pragma nv_exec_check_disable
template <int N, typename R, typename BA, typename KA>
NECG_HD bool term_value(const BA &b, const KA &kr, const Consts<N> &cs, R &ov, R &tau2, R &rho, R &sig) {
    R Bi[tri(N)], T[3 * N];
    const bool ok = term_core<N>(b, kr, Bi, T, ov);
    sig = term_sig<N>(cs, T);
    rho = coulomb_sum<N>(Bi, T, cs);
    tau2 = term_tau2<N>(b, kr, Bi, T);
    return ok;
}

// The bra gradient of one term's h and ov (Part<N> fields: dF/dA_k packed without
// its A_k^-1 part, that part's coefficient, dF/ds_k), in the direct formulation:
//   dh/dA_k = ov (-eta (1.5 Bi + D_k D_k^T) + Bi (6 N_l' + W) Bi + Q D_k^T + D_k Q^T
//                 + 0.75 eta A_k^-1),  dh/ds_k = 2 ov (A_k Q - eta Y),
//   D_k = S_k - T,  Y = A_k D_k = A_l' (T - S_l'),  Q = Bi (Z' - 4 A_l' M Y),
// and the same of ov with eta = 1 and without W, N_l' and Q.  The other side's N_l'
// stands where the sums' form (term_raw) has 6 M - 6 (M A_k Bi + Bi A_k M) + 6 Bi N_k Bi,
// which cancels when the bra is the tighter function; sums over a basis have that
// function's own term beside it, single elements do not.  Y is formed with the
// looser side, whose difference of positions does not cancel.
#pragma nv_exec_check_disable
template <int N, typename R, typename BA, typename KA>
NECG_HD bool term_grad(const BA &b, const KA &kr, const Consts<N> &cs, R (&gH)[tri(N) + 1 + 3 * N],
                       R (&gS)[tri(N) + 1 + 3 * N]) {
    using BL = BraLayout<N>;
    using KL = KetLayout<N>;
    constexpr int TR = tri(N);
    R Bi[TR], T[3 * N], ov;
    const bool ok = term_core<N>(b, kr, Bi, T, ov);
    R Z[3 * N], W[TR];  // 2 Z', 2 W
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) Z[t] = R(0.0);
#pragma unroll
    for (int t = 0; t < TR; ++t) W[t] = R(0.0);
    const R rho = coulomb_grad<N>(Bi, T, cs, Z, W);
    const R eta = term_tau2<N>(b, kr, Bi, T) + rho - term_sig<N>(cs, T);
    const bool use_l = kr[KL::tMA] <= b(BL::tMA);
    R Y[3 * N], p[3 * N];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R yk = R(0.0), yl = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                yk += b(BL::A + sx(i, k)) * (b(BL::S + 3 * k + c) - T[3 * k + c]);
                yl += kr[KL::Ap + sx(i, k)] * (T[3 * k + c] - kr[KL::Sp + 3 * k + c]);
            }
            Y[3 * i + c] = use_l ? yl : yk;
        }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += cs.M[i * N + k] * Y[3 * k + c];
            p[3 * i + c] = v;  // M Y
        }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        Z[3 * i + 2] -= cs.efs * cs.q[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += kr[KL::Ap + sx(i, k)] * p[3 * k + c];
            Z[3 * i + c] -= 8.0 * v;
        }
    }
    R Q[3 * N];  // 2 Q
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += Bi[sx(i, k)] * Z[3 * k + c];
            Q[3 * i + c] = v;
        }
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += b(BL::A + sx(i, k)) * Q[3 * k + c];
            const R y = 2.0 * (ov * Y[3 * i + c]);
            gH[TR + 1 + 3 * i + c] = ov * v - eta * y;
            gS[TR + 1 + 3 * i + c] = -y;
        }
#pragma unroll
    for (int t = 0; t < TR; ++t) W[t] = 0.5 * W[t] - 0.75 * kr[KL::Np8 + t];  // W + 6 N_l'
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) {
        T[t] = b(BL::S + t) - T[t];  // D_k
        Q[t] *= 0.5;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        R col[N];  // column j of (W + 6 N_l') Bi
#pragma unroll
        for (int a = 0; a < N; ++a) {
            R v = W[sx(a, 0)] * Bi[sx(0, j)];
#pragma unroll
            for (int k = 1; k < N; ++k) v += W[sx(a, k)] * Bi[sx(k, j)];
            col[a] = v;
        }
#pragma unroll
        for (int i = j; i < N; ++i) {
            R v = R(0.0), u = 1.5 * Bi[sx(i, j)];
#pragma unroll
            for (int a = 0; a < N; ++a) v += Bi[sx(i, a)] * col[a];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v += Q[3 * i + c] * T[3 * j + c] + T[3 * i + c] * Q[3 * j + c];
                u += T[3 * i + c] * T[3 * j + c];
            }
            gH[sx(i, j)] = ov * (v - eta * u);
            gS[sx(i, j)] = -(ov * u);
        }
    }
    gH[TR] = 0.75 * (ov * eta);
    gS[TR] = 0.75 * ov;
    return ok;
}

// f(integral_constant<int, I>) for I = A .. END - 1, unrolled
template <int I> struct IntC {
    static constexpr int value = I;
};
template <int A, int END, typename F> NECG_HD void unrolled(F &&f) {
    if constexpr (A < END) {
        f(IntC<A>{});
        unrolled<A + 1, END>(f);
    }
}

// Fields of the raw sums of one basis function (Part<N>::size of them, the same
// count and order as the partial buffers): G[tri] (derivative with respect to
// A through B and e), one scalar, g[3N] (derivative with respect to e).  Raw values of
// one term for side s, before the weight w ov:
//   H:  X = 2 (Bi (6 N + W) Bi - Q D_s^T - D_s Q^T - eta U_s),  2 eta,  2 (Q + eta D_s)
//   S:  -U_s,                                                   1,      D_s
// so that H - 2 E S holds twice the G, twice the scalar and once the g of the
// gradient of h - E ov.  term_raw hands the fields out in pairs, for outputs
// that combine two values at a time: pair i < tri holds G_i and g_i, the
// remaining g follow two by two, and the scalar comes with the last g when
// their number is odd, alone otherwise (n <= 5, where tri <= 3 n).
template <int N> struct RawPairs {
    static constexpr int T = tri(N), V = 3 * N;
    static constexpr int lead = T < V ? T : V;
    static constexpr int left = V - lead;
    static constexpr bool odd = left & 1;               // the scalar's pair also holds g[V - 1]
    static constexpr int count = lead + left / 2 + 1;   // the last one holds the scalar
    static constexpr int scalar = T;                    // its field index
    // pair and side (0, 1) of field f
    __host__ __device__ static constexpr int pair_of(int f) {
        return f < T ? f : f == T ? count - 1 : f - T - 1 < lead ? f - T - 1 : lead + (f - T - 1 - lead) / 2;
    }
    // fields of pair i
    __host__ __device__ static constexpr int fa(int i) { return i < lead ? i : T + 1 + lead + 2 * (i - lead); }
    __host__ __device__ static constexpr int fb(int i) {
        return i < lead ? T + 1 + i : odd && i == count - 1 ? scalar : fa(i) + 1;
    }
    static constexpr int paired = odd ? count : count - 1;  // pairs with two fields
    __host__ __device__ static constexpr int side_of(int f) {
        return f < T ? 0 : f == T ? (odd ? 1 : 0) : f - T - 1 < lead ? 1 : (f - T - 1 - lead) & 1;
    }
};

// The raw values of one side (KET: the ket's) handed to `out`, pair by pair.
template <int N, bool KET, int I, typename R, typename OUT> NECG_HD void put_s(OUT &out, R va, R vb) {
    if constexpr (KET) out.template sk<I>(va, vb);
    else out.template sb<I>(va, vb);
}
template <int N, bool KET, int I, typename R, typename OUT> NECG_HD void put_h(OUT &out, R va, R vb) {
    if constexpr (KET) out.template hk<I>(va, vb);
    else out.template hb<I>(va, vb);
}
// S: -U = -(1.5 Bi + D D^T), D, 1
#pragma nv_exec_check_disable
template <int N, bool KET, typename R, typename OUT>
NECG_HD void raw_s(const R (&Bi)[tri(N)], const R (&D)[3 * N], OUT &out) {
    using RP = RawPairs<N>;
    unrolled<0, N>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        unrolled<0, i + 1>([&](auto jc) {
            constexpr int j = decltype(jc)::value, t = sx(i, j);
            R u = 1.5 * Bi[t];
#pragma unroll
            for (int c = 0; c < 3; ++c) u += D[3 * i + c] * D[3 * j + c];
            if constexpr (t < RP::lead) put_s<N, KET, t, R>(out, -u, D[t]);
            else if constexpr (!KET) out.sb1(t, -u);
        });
    });
    unrolled<0, RP::left / 2>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        put_s<N, KET, RP::lead + q, R>(out, D[RP::lead + 2 * q], D[RP::lead + 2 * q + 1]);
    });
    if constexpr (RP::odd) put_s<N, KET, RP::count - 1, R>(out, D[3 * N - 1], R(1.0));
}
// H's entry (i, j): x = (Bi W Bi - 1.5 et Bi)_ij less Q' D^T + D Q'^T, and its g = Q' + et D / 2
#pragma nv_exec_check_disable
template <int N, bool KET, int I, int J, typename R, typename OUT>
NECG_HD void raw_h(R x, const R (&D)[3 * N], const R (&Q)[3 * N], R eh, OUT &out) {
    constexpr int t = sx(I, J);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        x -= Q[3 * I + c] * D[3 * J + c];
        x -= D[3 * I + c] * Q[3 * J + c];
    }
    if constexpr (t < RawPairs<N>::lead) put_h<N, KET, t, R>(out, x, Q[t] + eh * D[t]);
    else if constexpr (!KET) out.hb1(t, x);
}
// the remaining g
#pragma nv_exec_check_disable
template <int N, bool KET, typename R, typename OUT>
NECG_HD void raw_h_rest(const R (&D)[3 * N], const R (&Q)[3 * N], R eh, R et, OUT &out) {
    using RP = RawPairs<N>;
    unrolled<0, RP::left / 2>([&](auto qc) {
        constexpr int q = decltype(qc)::value, u = RP::lead + 2 * q;
        put_h<N, KET, RP::lead + q, R>(out, Q[u] + eh * D[u], Q[u + 1] + eh * D[u + 1]);
    });
    if constexpr (RP::odd) put_h<N, KET, RP::count - 1, R>(out, Q[3 * N - 1] + eh * D[3 * N - 1], et);
}
// all of one side's H values from X = Bi W Bi - 1.5 et Bi and Q
#pragma nv_exec_check_disable
template <int N, bool KET, typename R, typename OUT>
NECG_HD void raw_h_side(const R (&X)[tri(N)], const R (&D)[3 * N], const R (&Q)[3 * N], R eh, R et, OUT &out) {
    R Qs[3 * N];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) Qs[t] = Q[t] + eh * D[t];
    unrolled<0, N>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        unrolled<0, i + 1>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            raw_h<N, KET, i, j, R>(X[sx(i, j)], D, Qs, eh, out);
        });
    });
    raw_h_rest<N, KET, R>(D, Qs, eh, et, out);
}
// One (k, l, P) term: the overlap and the raw values above, handed to `out`:
//   out.begin(ov)              once, first
//   out.sb<i>(va, vb), sk<i>   pair i of the bra's / the ket's S values
//   out.hb<i>(va, vb), hk<i>   pair i of the bra's / the ket's H values, with eta - E2 / 2
//                              in the place of eta (E2 = 2 E gives the gradient of h - E ov)
//   out.scalar(eta2)           the scalar pair when it holds nothing else
//   out.sb1 / out.hb1(f, v)    single fields (n = 6 only, which has no ket side)
// OUT::kets: the ket's values are wanted; OUT::ket_s: its S values too.
// eta2_out = 2 eta (so h = ov eta2_out / 2).  The S values leave before the
// Coulomb sum, so that U is not live across it, and D_k and D_l are formed again
// after it for the same reason.  One side's values leave after the other's: side by
// side saves a few operations and costs registers (LiH K = 1024 on a B200: 2.50 ms,
// 2.52 with H's and 2.53 with S's two sides in one loop).
#pragma nv_exec_check_disable
template <int N, typename R, typename BA, typename KA, typename OUT>
NECG_HD bool term_raw(const BA &b, const KA &kr, const Consts<N> &cs, R E2, OUT &out, R &eta2_out, R &ov_out) {
    using BL = BraLayout<N>;
    using KL = KetLayout<N>;
    using RP = RawPairs<N>;
    constexpr int TR = tri(N), V = 3 * N;
    R Bi[TR], T[V], ov;
    const bool ok = term_core<N>(b, kr, Bi, T, ov);
    ov_out = ov;
    out.begin(ov);
    if constexpr (OUT::ket_s) {
        R D[V];
#pragma unroll
        for (int t = 0; t < V; ++t) D[t] = T[t] - kr[KL::Sp + t];
        raw_s<N, true, R>(Bi, D, out);
    }
    // tau and the bra's part of Q's right-hand side: V8 = -8 N D, D = D_k;
    // 4 tau = 12 tr(M A_s) + 1.5 <-8 N_s, Bi> + <D, V8>.  The trace cancels for the
    // tighter side (term_tau2), so it is formed with both and the one of the
    // smaller tr(M A) taken: tri(N) products more, where selecting N_s would take
    // twice as many instructions.
    R Z[V], W[TR], eta2;
    {
        R D[V];
#pragma unroll
        for (int t = 0; t < V; ++t) D[t] = T[t] - b(BL::S + t);
        raw_s<N, false, R>(Bi, D, out);
        R dg = R(0.0), od = R(0.0), dl = R(0.0), ol = R(0.0);
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int k = 0; k <= i; ++k) {
                // each element of N is read once and used for the three columns
                const R a = b(BL::N8 + sx(i, k)), al = kr[KL::Np8 + sx(i, k)];
                W[sx(i, k)] = -1.5 * a;
                if (i == k) {
                    dg = (i == 0) ? a * Bi[0] : dg + a * Bi[sx(i, k)];
                    dl = (i == 0) ? al * Bi[0] : dl + al * Bi[sx(i, k)];
                } else {
                    od = (i == 1) ? a * Bi[sx(1, 0)] : od + a * Bi[sx(i, k)];
                    ol = (i == 1) ? al * Bi[sx(1, 0)] : ol + al * Bi[sx(i, k)];
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    // element (i, k) is the first of row i when k = 0, and the first of row k when i = k = 0
                    if (k == 0)
                        Z[3 * i + c] = a * D[c];
                    else
                        Z[3 * i + c] += a * D[3 * k + c];
                    if (k < i) Z[3 * k + c] += a * D[3 * i + c];
                }
            }
        R e0 = D[0] * Z[0], e1 = D[1] * Z[1], e2 = D[2] * Z[2];
#pragma unroll
        for (int i = 1; i < N; ++i) {
            e0 += D[3 * i] * Z[3 * i];
            e1 += D[3 * i + 1] * Z[3 * i + 1];
            e2 += D[3 * i + 2] * Z[3 * i + 2];
        }
        const R tl = kr[KL::tMA], tk = b(BL::tMA);
        const R xk = 8.0 * tk + (dg + 2.0 * od), xl = 8.0 * tl + (dl + 2.0 * ol);  // 8 tr(M X), of either side
        eta2 = 1.5 * (tl <= tk ? xl : xk) + (e0 + e1 + e2);
    }
    {
        R sg = R(0.0);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const R eq = cs.efs * cs.q[i];
            sg = (i == 0) ? eq * T[2] : sg + eq * T[3 * i + 2];
            Z[3 * i + 2] -= eq;
        }
        eta2 -= 2.0 * sg;
    }
    const R rho = coulomb_grad<N>(Bi, T, cs, Z, W);
    eta2 += 2.0 * rho;
    eta2_out = eta2;
    const R et = eta2 - E2, eh = 0.5 * et, e15 = 1.5 * et;
    if (!RP::odd) out.scalar(et);
    // X = Bi W Bi - 1.5 et Bi - Q' D^T - D Q'^T with Q' = Q + et D / 2 (the D D^T
    // part of et U folded into the outer products); g = Q' + et D / 2.  Up to the
    // outer products it is the same for both sides.
    R Q[V];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R s = Bi[sx(i, 0)] * Z[c];
#pragma unroll
            for (int k = 1; k < N; ++k) s += Bi[sx(i, k)] * Z[3 * k + c];
            Q[3 * i + c] = s;
        }
    R X[TR];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        R col[N];  // column j of W Bi
#pragma unroll
        for (int a = 0; a < N; ++a) {
            R s = W[sx(a, 0)] * Bi[sx(0, j)];
#pragma unroll
            for (int k = 1; k < N; ++k) s += W[sx(a, k)] * Bi[sx(k, j)];
            col[a] = s;
        }
#pragma unroll
        for (int i = j; i < N; ++i) {
            R s = -(e15 * Bi[sx(i, j)]);
#pragma unroll
            for (int a = 0; a < N; ++a) s += Bi[sx(i, a)] * col[a];
            X[sx(i, j)] = s;
        }
    }
    {
        R D[V];
#pragma unroll
        for (int t = 0; t < V; ++t) D[t] = T[t] - b(BL::S + t);
        raw_h_side<N, false, R>(X, D, Q, eh, et, out);
    }
    if constexpr (OUT::kets) {
        R D[V];
#pragma unroll
        for (int t = 0; t < V; ++t) D[t] = T[t] - kr[KL::Sp + t];
        raw_h_side<N, true, R>(X, D, Q, eh, et, out);
    }
    return ok;
}

// The gradient of one side from its raw sums r (H, 2 S, or their combination H - 2 E
// S) and its A, in the frame of the sums: dF/dA = r_G / 2 + 0.75 F A^-1, F = r_scalar /
// 2, and dF/ds = A r_g.  o: Part<N> fields.
#pragma nv_exec_check_disable
template <int N, typename R, typename RAW, typename FA>
NECG_HD void fold_raw(const RAW &r, const FA &A, R (&o)[tri(N) + 1 + 3 * N]) {
    constexpr int TR = tri(N);
#pragma unroll
    for (int t = 0; t < TR; ++t) o[t] = 0.5 * r(t);
    o[TR] = 0.375 * r(TR);
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = A(sx(i, 0)) * r(TR + 1 + c);
#pragma unroll
            for (int k = 1; k < N; ++k) v += A(sx(i, k)) * r(TR + 1 + 3 * k + c);
            o[TR + 1 + 3 * i + c] = v;
        }
}

// The bra's explicit share of dh through tau, added to its combined raw sums r:
// tau depends on A_k and s_k directly (not through B and e).  With the bra's raw S
// sums s = (-U_k, 1, D_k)
//   dh/dA_k += 2 (3 M s_1 + 2 (M A s_U + s_U A M)),   dh/de_k += 8 M A s_D
// (r's G is held twice).
#pragma nv_exec_check_disable
template <int N, typename R, typename SRAW, typename FA>
NECG_HD void explicit_tau(const SRAW &sr, const FA &A, const Consts<N> &cs, R (&r)[tri(N) + 1 + 3 * N]) {
    constexpr int TR = tri(N);
    const R s1 = sr(TR);
    R y[3 * N], MA[N * N];  // A s_D, M A
#pragma unroll
    for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += A(sx(i, k)) * sr(TR + 1 + 3 * k + c);
            y[3 * i + c] = v;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += cs.M[i * N + k] * A(sx(k, j));
            MA[i * N + j] = v;
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R v = R(0.0);
#pragma unroll
            for (int k = 0; k < N; ++k) v += cs.M[i * N + k] * y[3 * k + c];
            r[TR + 1 + 3 * i + c] += 8.0 * v;
        }
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            R v = 3.0 * cs.M[i * N + j] * s1;
#pragma unroll
            for (int k = 0; k < N; ++k)
                v += 2.0 * (MA[i * N + k] * sr(sx(k, j)) + sr(sx(i, k)) * MA[j * N + k]);
            r[sx(i, j)] += 4.0 * v;
        }
    }
}

// One side's fields in an array, read as a functor.
template <typename R> struct FieldsOf {
    const R *p;
    NECG_HD const R &operator()(int f) const { return p[f]; }
};

// One term of the dipole element of python/rrms.py:21-120 for the bra record
// (k, Pe) and the ket record (l, P) (both in KetLayout: symmetry applied to both
// sides): B = A_k'' + A_l', T = Bi (A_k'' s_k'' + A_l' s_l') (rrms's st), and
// ov = sqrt(8^n) (|L_k| |L_l| / |B|)^{3/2} exp(<e, T> - i1 - i2).  rrms returns
// (ov, T[n1] ov).  Returns false if B is not positive definite.
#pragma nv_exec_check_disable
template <int N, typename R, typename KA, typename KB>
NECG_HD bool term_dipole(const KA &kb, const KB &kr, const Consts<N> &cs, R (&T)[3 * N], R &ov) {
    using KL = KetLayout<N>;
    R Bi[tri(N)], m32;
    bool ok;
    {
        R B[tri(N)];
#pragma unroll
        for (int t = 0; t < tri(N); ++t) B[t] = kb[KL::Ap + t] + kr[KL::Ap + t];
        ok = spd_inverse<N>(B, Bi, m32);
    }
    R e[3 * N];
#pragma unroll
    for (int t = 0; t < 3 * N; ++t) e[t] = kb[KL::ASp + t] + kr[KL::ASp + t];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R s = Bi[sx(i, 0)] * e[c];
#pragma unroll
            for (int k = 1; k < N; ++k) s += Bi[sx(i, k)] * e[3 * k + c];
            T[3 * i + c] = s;
        }
    R i3 = e[0] * T[0];
#pragma unroll
    for (int t = 1; t < 3 * N; ++t) i3 += e[t] * T[t];
    ov = cs.sqrt8n * kb[KL::pre] * kr[KL::pre] * m32 * exp(i3 - kb[KL::i2] - kr[KL::i2]);
    return ok;
}

}  // namespace necg
