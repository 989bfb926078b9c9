// necg_capi.cu -- the extern "C" boundary declared in include/necg.h.
//
// A handle owns one particle system's constants (mass, charges, symmetry set)
// on the device plus the workspace one evaluation needs for bases of up to
// K_max functions:
//   bra   BraLayout<n>::size * K_max       per-basis data (K_max rounded up to 32)
//   ket   KetLayout<n>::size * K_max * nst per-(l, P) ket records
//   part  part_doubles(n, K_max)           tile partials of the ordered gradient, or
//                                          the symmetric passes' per-basis sums
//   H, S  K_max^2 each (used when the caller passes no H/S)
//   rows  2 K_max, scal 4, x/g staging for the host-pointer entry point
// The tile lists and the partial buffers of the symmetric passes, whose sizes follow
// from K and the settings, are made when a call first needs them (as are the dipole's
// classes and the host entry point's pinned buffer): every device-pointer entry
// point is stream-ordered, and capturable in a CUDA graph once a call with the same
// K and settings has run.
//
// Handle memory comes from one stream-ordered pool per device (cudaMemPool_t,
// blocks kept for reuse), allocated and freed on the library's own
// non-blocking stream of that device, or on the caller's stream when an
// evaluation grows a buffer.  Unlike cudaMalloc / cudaFree, creating and
// destroying a handle then never waits for work that other streams have in
// flight, so a server can admit and retire runs while its steps keep running.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "necg_handle.h"
#include "necg_kernels.cuh"
#include "necg_maps.h"
#include "necg_math.cuh"
#include "necg_trace.h"

using necg::LaunchArgs;

namespace {

// Doubles before g in a handle's output block: f, the two status words, padding.
constexpr size_t kOutHead = 4;

// Status code of the two device status words (flags, first failing pair).
int status_code(const int st[2], long long *bad_pair) {
    if (bad_pair) *bad_pair = st[1] == 0x7fffffff ? -1 : (long long)st[1];
    if (st[0] & 1) return NECG_ERR_NOT_PD;
    if (st[0] & 2) return NECG_ERR_NONFINITE;
    if (st[0] & 4) return NECG_ERR_ARG;
    return NECG_OK;
}

int cuda_fail(cudaError_t e) {
    if (e == cudaSuccess) return NECG_OK;
    return e == cudaErrorMemoryAllocation ? NECG_ERR_ALLOC : NECG_ERR_CUDA;
}

#define CK(x)                                  \
    do {                                       \
        cudaError_t _e = (x);                  \
        if (_e != cudaSuccess) return cuda_fail(_e); \
    } while (0)

// The per-device pool and stream, made on first use with that device current.
struct DevicePool {
    std::once_flag once;
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    cudaError_t err = cudaSuccess;
};
DevicePool g_pools[64];

cudaError_t device_pool(int dev, cudaMemPool_t *pool, cudaStream_t *stream) {
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    DevicePool &d = g_pools[dev];
    std::call_once(d.once, [&] {
        cudaMemPoolProps props;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        d.err = cudaMemPoolCreate(&d.pool, &props);
        if (d.err == cudaSuccess) {
            uint64_t keep = UINT64_MAX;  // freed blocks stay in the pool for the next handle
            d.err = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        if (d.err == cudaSuccess) d.err = cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking);
    });
    *pool = d.pool;
    *stream = d.stream;
    return d.err;
}

// Stream-ordered allocation from the handle's device pool on stream st (the
// library stream when st is null).
template <typename T> cudaError_t pool_alloc(necg_handle *h, T **p, size_t bytes, cudaStream_t st = nullptr) {
    cudaMemPool_t pool;
    cudaStream_t ls;
    cudaError_t e = device_pool(h->device, &pool, &ls);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void **)p, bytes, pool, st ? st : ls);
    if (e != cudaSuccess) *p = nullptr;
    return e;
}

void pool_free(necg_handle *h, void *p, cudaStream_t st = nullptr) {
    if (!p) return;
    cudaMemPool_t pool;
    cudaStream_t ls;
    if (device_pool(h->device, &pool, &ls) == cudaSuccess) cudaFreeAsync(p, st ? st : ls);
}

cudaStream_t lib_stream(necg_handle *h) {
    cudaMemPool_t pool;
    cudaStream_t ls = nullptr;
    device_pool(h->device, &pool, &ls);
    return ls;
}

template <typename T> int dalloc(necg_handle *h, T **p, size_t count) {
    size_t bytes = count * sizeof(T);
    if (bytes == 0) bytes = 16;
    cudaError_t e = pool_alloc(h, p, bytes);
    if (e != cudaSuccess) return cuda_fail(e);
    h->ws_bytes += (long long)bytes;
    return NECG_OK;
}

// Phase event i of the evaluation (profiling).  While the stream is being
// captured it is recorded as an external event, so that the captured graph
// records it when it runs.
void mark(necg_handle *h, int i, cudaStream_t st) {
    if (!h->profile) return;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cap);
    if (cap == cudaStreamCaptureStatusActive) cudaEventRecordWithFlags(h->ev[i], st, cudaEventRecordExternal);
    else cudaEventRecord(h->ev[i], st);
}

void free_all(necg_handle *h) {
    for (cudaEvent_t &e : h->ev)
        if (e) cudaEventDestroy(e);
    void *ptrs[] = {h->d_sml, h->d_sms, h->d_scvv, h->d_bra, h->d_ket, h->d_part, h->d_H,
                    h->d_S, h->d_rows, h->d_scal, h->d_x, h->d_out,
                    h->d_tiles, h->d_pinv, h->d_kcnt, h->d_ksrc, h->d_kcoef, h->d_lists,
                    h->d_psym, h->d_qcount, h->d_Hp, h->d_Sp, h->d_xsym, h->d_dipcls};
    for (void *p : ptrs) pool_free(h, p);
}

// Lists and buffers change only outside a stream capture (their allocations would
// belong to the captured graph, and the lists would not be there before a replay).
bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
}
int not_capturing(cudaStream_t st) { return capturing(st) ? NECG_ERR_CUDA : NECG_OK; }

// Make one of the handle's buffers hold `need` entries, or (exact) just those.
template <typename T> int fit(necg_handle *h, T **p, size_t *cap, size_t need, cudaStream_t st, bool exact = false) {
    if (exact ? need == *cap : need <= *cap) return NECG_OK;
    pool_free(h, *p, st);
    *p = nullptr;
    h->ws_bytes -= (long long)(*cap * sizeof(T));
    *cap = 0;
    ++h->gversion;  // buffers and lists a captured graph may hold changed
    if (!need) return NECG_OK;
    CK(pool_alloc(h, p, need * sizeof(T), st));
    h->ws_bytes += (long long)(need * sizeof(T));
    *cap = need;
    return NECG_OK;
}

// Energy tiles over the lower triangle: (kb, lc) with lc * LC <= row_last(K, kb).
int ensure_tiles(necg_handle *h, int K, cudaStream_t st) {
    if (h->tiles_K == K && h->tiles_lc == h->lc_e) return NECG_OK;
    int rc = not_capturing(st);
    if (rc) return rc;
    const int nt = necg::tiles_before(K, h->lc_e, necg::row_blocks(K));
    h->tiles_K = -1;
    if ((rc = fit(h, &h->d_tiles, &h->tiles_cap, (size_t)nt, st))) return rc;
    necg::launch_tile_list(h->d_tiles, K, h->lc_e, st);
    CK(cudaGetLastError());
    h->tiles_K = K;
    ++h->gversion;  // buffers and lists a captured graph may hold changed
    h->tiles_lc = h->lc_e;
    h->ntiles = nt;
    return NECG_OK;
}

// The K x K buffers of a fused pass with split terms whose caller wants H and S.
int ensure_split_matrices(necg_handle *h, int K, int npc, cudaStream_t st) {
    const size_t need = npc > 1 ? (size_t)npc * K * K : 0;
    if (need <= h->hp_cap) return NECG_OK;
    int rc = not_capturing(st);
    if (rc) return rc;
    size_t cap = h->hp_cap;
    if ((rc = fit(h, &h->d_Hp, &cap, need, st))) h->hp_cap = 0;
    else rc = fit(h, &h->d_Sp, &h->hp_cap, need, st);
    return rc;
}

// Lower-triangle tiles of chunk LC for the symmetric passes and the queue of the
// block variants (necg_tiles.h), and the partial buffers for this K and LC with npc
// slots per tile.  Settings that have changed since the lists were made give back what
// they need less (while the lists stay as they are, so do the buffers: a caller's own
// captured graphs hold them).
int ensure_sym_tiles(necg_handle *h, int K, cudaStream_t st, int npc) {
    const int PB = necg::part_stride(h->n) + 1, LC = h->lc_s;
    const int gw = necg::fused_block_warps(h->minb_s);  // tiles per group of the block variants
    const bool same = h->stiles_K == K && h->stiles_lc == LC && h->sgroups_w == gw;
    if (same && (size_t)h->nstiles * PB * (32 + LC) * 2 * npc <= h->psym_cap) return NECG_OK;
    const bool exact = !same && h->refit;
    int rc = not_capturing(st);
    if (rc) return rc;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    const necg::SymQueue q = necg::sym_queue(K, LC, gw, h->nst, sms);
    const size_t xneed = q.ntail ? (size_t)q.ntail * gw * (q.parts - 1) * necg::fsym_tail_slot(PB, LC) : 0;
    if ((rc = fit(h, &h->d_psym, &h->psym_cap, (size_t)q.ntiles * PB * (32 + LC) * 2 * npc, st, exact))) return rc;
    if ((rc = fit(h, &h->d_xsym, &h->xsym_cap, xneed, st, exact))) return rc;
    if (exact && h->hp_cap) {  // ensure_split_matrices makes them again if they are wanted
        size_t cap = h->hp_cap;
        fit(h, &h->d_Hp, &cap, 0, st, true);
        fit(h, &h->d_Sp, &h->hp_cap, 0, st, true);
    }
    if (same) return NECG_OK;
    // one buffer for all lists: the int2 lists, then the int lists
    const int nkb = necg::row_blocks(K), nb = necg::groups_before(K, LC, 8, -1), nu = q.units();
    const size_t n2 = (size_t)q.ntiles + nu + nb + 2 * nkb, need = n2 + (q.ntiles + nkb + 1 + 1) / 2;
    h->stiles_K = -1;
    if ((rc = fit(h, &h->d_lists, &h->lists_cap, need, st, exact))) return rc;
    h->refit = false;
    if (!h->d_qcount) CK(pool_alloc(h, &h->d_qcount, sizeof(int), st));
    necg::SymLists &o = h->lists;
    o.tiles = h->d_lists;
    o.groups = o.tiles + q.ntiles;
    o.bgroups = o.groups + nu;
    o.urange = o.bgroups + nb;
    o.burange = o.urange + nkb;
    o.tslot = (int *)(o.burange + nkb);
    o.start = o.tslot + q.ntiles;
    necg::launch_sym_lists(q, o, st);
    CK(cudaGetLastError());
    h->queue = q;
    h->nbgroups = nb;
    h->nstiles = q.ntiles;
    h->sgroups_w = gw;
    h->stiles_lc = LC;
    h->stiles_K = K;
    ++h->gversion;
    return NECG_OK;
}

}  // namespace

int necg::prepare_fused(necg_handle *h, int K, cudaStream_t st) {
    if (!h || !h->sym_ok) return NECG_ERR_UNSUPPORTED;
    CK(cudaSetDevice(h->device));
    return ensure_sym_tiles(h, K, st, fused_splits(h));
}

namespace {

// Inverse of each symmetry term (sml and sms both inverted) and the map of a
// ket gradient from P's frame to the basis function's frame.  Sets sym_ok
// when every term's inverse is in the set and n <= 5.
int setup_symmetric(necg_handle *h) {
    const int n = h->n, nst = h->nst;
    if (n > 5) return NECG_OK;
    std::vector<int> pinv;
    if (!necg::inverse_terms(n, nst, h->sml.data(), h->sms.data(), pinv)) return NECG_OK;  // ordered pass only
    const necg::RawMapTable t = necg::raw_map_table(n, nst, h->sml.data(), h->sms.data(), necg::ket_slots(n),
                                                    [n](int f) { return necg::ket_slot(n, f); });
    int rc = NECG_OK;
    if (!rc) rc = dalloc(h, &h->d_pinv, (size_t)nst);
    if (!rc) rc = dalloc(h, &h->d_kcnt, t.cnt.size());
    if (!rc) rc = dalloc(h, &h->d_ksrc, t.src.size());
    if (!rc) rc = dalloc(h, &h->d_kcoef, t.coef.size());
    if (rc) return rc;
    cudaStream_t ls = lib_stream(h);
    CK(cudaMemcpyAsync(h->d_pinv, pinv.data(), nst * sizeof(int), cudaMemcpyHostToDevice, ls));
    CK(cudaMemcpyAsync(h->d_kcnt, t.cnt.data(), t.cnt.size() * sizeof(int), cudaMemcpyHostToDevice, ls));
    CK(cudaMemcpyAsync(h->d_ksrc, t.src.data(), t.src.size() * sizeof(int), cudaMemcpyHostToDevice, ls));
    CK(cudaMemcpyAsync(h->d_kcoef, t.coef.data(), t.coef.size() * sizeof(double), cudaMemcpyHostToDevice, ls));
    CK(cudaStreamSynchronize(ls));  // the host vectors above end with this scope
    h->kmaxnz = t.maxnz;
    h->kfold = t.fold;
    h->sym_ok = true;
    h->grad_mode = 1;
    return NECG_OK;
}

// Classes of the dipole's nst^2 terms (Pe, P) of a pair (dipole_group_kernel):
// Q = P Pe^-1, when every Q is in the set and the shift maps follow the
// coordinate maps (sms = kron(sml^-1, I3), which also gives Pe^-1).  Larger sets
// than 128 terms keep the general path (the search for Q grows as nst^3).
// Set up by the handle's first dipole outside a stream capture (it allocates and
// waits; until then the general path runs).
int setup_dipole(necg_handle *h, cudaStream_t st) {
    const int n = h->n, nst = h->nst, m = 3 * n, nn = n * n;
    if (h->dip_ready) return NECG_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(st, &cap));
    if (cap != cudaStreamCaptureStatusNone) return NECG_OK;
    h->dip_ready = true;
    if (nst < 2 || nst > 128) return NECG_OK;
    std::vector<double> inv((size_t)nst * nn);
    for (int p = 0; p < nst; ++p) {
        const double *S = &h->sms[(size_t)p * m * m], *P = &h->sml[(size_t)p * nn];
        double *I = &inv[(size_t)p * nn];
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) I[i * n + j] = S[(3 * i) * m + 3 * j];
        for (int r = 0; r < m; ++r)  // sms = kron(I, I3) ...
            for (int c = 0; c < m; ++c)
                if (fabs(S[r * m + c] - (r % 3 == c % 3 ? I[(r / 3) * n + c / 3] : 0.0)) > 1e-12) return NECG_OK;
        for (int i = 0; i < n; ++i)  // ... and I = P^-1
            for (int j = 0; j < n; ++j) {
                double v = 0.0;
                for (int k = 0; k < n; ++k) v += I[i * n + k] * P[k * n + j];
                if (fabs(v - (i == j ? 1.0 : 0.0)) > 1e-12) return NECG_OK;
            }
    }
    std::vector<double> cls((size_t)nst * (nn + 1), 0.0), Q(nn);
    for (int pe = 0; pe < nst; ++pe)
        for (int p = 0; p < nst; ++p) {
            for (int i = 0; i < n; ++i)
                for (int j = 0; j < n; ++j) {
                    double v = 0.0;
                    for (int k = 0; k < n; ++k) v += h->sml[(size_t)p * nn + i * n + k] * inv[(size_t)pe * nn + k * n + j];
                    Q[i * n + j] = v;
                }
            int q = 0;
            for (; q < nst; ++q) {
                bool same = true;
                for (int x = 0; x < nn && same; ++x) same = fabs(Q[x] - h->sml[(size_t)q * nn + x]) < 1e-12;
                if (same) break;
            }
            if (q == nst) return NECG_OK;  // not closed under products
            double *c = &cls[(size_t)q * (nn + 1)];
            const double w = h->scvv[pe] * h->scvv[p];
            c[0] += w;
            for (int x = 0; x < nn; ++x) c[1 + x] += w * inv[(size_t)pe * nn + x];
        }
    int rc = dalloc(h, &h->d_dipcls, cls.size());
    if (rc) return rc;
    cudaStream_t ls = lib_stream(h);
    CK(cudaMemcpyAsync(h->d_dipcls, cls.data(), cls.size() * sizeof(double), cudaMemcpyHostToDevice, ls));
    CK(cudaStreamSynchronize(ls));  // cls ends with this scope
    return NECG_OK;
}

LaunchArgs base_args(necg_handle *h, int K) {
    LaunchArgs a;
    memset(&a, 0, sizeof(a));
    a.n = h->n;
    a.K = K;
    a.nst = h->nst;
    a.efs = h->efs;
    a.mass_h = h->mass.data();
    a.ncv_h = h->ncv.data();
    a.sml = h->d_sml;
    a.sms = h->d_sms;
    a.scvv = h->d_scvv;
    a.bra = h->d_bra;
    a.ket = h->d_ket;
    a.tiles = h->d_tiles;
    a.ntiles = h->ntiles;
    a.LC_e = h->lc_e;
    a.LC_g = h->lc_g;
    a.minb_e = h->minb_e;
    a.minb_g = h->minb_g;
    a.rows = h->d_rows;
    a.scal = h->d_scal;
    a.part = h->d_part;
    a.status = h->d_status;
    a.lam = 1.0;
    a.pinv = h->d_pinv;
    a.kmap = necg::RawMap{h->d_kcnt, h->d_ksrc, h->d_kcoef, h->kmaxnz, h->kfold};
    a.minb_s = h->minb_s;
    a.dip_cls = h->d_dipcls;
    a.sms_general = h->sms_general ? 1 : 0;
    return a;
}

// The tile lists and buffers of the symmetric passes, as ensure_sym_tiles left them.
void sym_args(const necg_handle *h, LaunchArgs &a) {
    a.stiles = h->lists.tiles;
    a.stile_start = h->lists.start;
    a.nstiles = h->nstiles;
    a.LC_s = h->lc_s;
    a.psym = h->d_psym;
    a.sgroups = h->lists.groups;
    a.nsgroups = h->queue.units();
    a.qcount = h->d_qcount;
    a.xsym = h->d_xsym;
    a.sg_tail0 = h->queue.tail0;
    a.sg_ntail = h->queue.ntail;
    a.sg_parts = h->queue.parts;
    a.urange = h->lists.urange;
    a.tslot = h->lists.tslot;
}

// The gradient passes after E and norm are in scal: symmetric (unordered pairs)
// when available, ordered otherwise.  (Mode 2 fuses the symmetric pass with the
// energy pass of necg_outprod; here H and S are already known, so the
// symmetric pass alone is used.)
int launch_gradient(necg_handle *h, LaunchArgs &a, cudaStream_t st) {
    if (h->grad_mode >= 1) {
        int rc = ensure_sym_tiles(h, a.K, st, 1);
        if (rc) return rc;
        sym_args(h, a);
        mark(h, 3, st);
        necg::launch_gsym(a, st);
        mark(h, 4, st);
        necg::launch_gsym_reduce(a, st);
        mark(h, 5, st);
        return NECG_OK;
    }
    mark(h, 3, st);
    necg::launch_grad_tiles(a, st);
    mark(h, 4, st);
    necg::launch_grad_reduce(a, st);
    mark(h, 5, st);
    return NECG_OK;
}

int check_K(necg_handle *h, int K) {
    if (!h) return NECG_ERR_ARG;
    if (K < 1) return NECG_ERR_ARG;
    if (K > h->K_max) return NECG_ERR_CAPACITY;
    return NECG_OK;
}

int begin(necg_handle *h, cudaStream_t st) {
    CK(cudaSetDevice(h->device));
    h->last_stream = st;  // the entry point's prep resets the status words
    return NECG_OK;
}

int finish_launch() {
    cudaError_t e = cudaGetLastError();
    return cuda_fail(e);
}

// The fused evaluation's launch sequence, from the records to the gradient,
// enqueued on st (no host synchronisation, so it can be captured).
int enqueue_fused(necg_handle *h, LaunchArgs &a, double *f_dev, double *g_dev, size_t siv, cudaStream_t st) {
    mark(h, 0, st);
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    mark(h, 1, st);
    if (necg::launch_fsym(a, st)) return NECG_ERR_ARG;
    if (necg::launch_fsym_tail(a, st)) return NECG_ERR_ARG;
    if (necg::launch_hs_reduce(a, st)) return NECG_ERR_ARG;
    mark(h, 2, st);
    mark(h, 3, st);
    if (necg::launch_fsym_sum(a, st)) return NECG_ERR_ARG;
    mark(h, 4, st);
    if (necg::launch_fsym_finish(a, f_dev, g_dev + siv, true, st)) return NECG_ERR_ARG;
    mark(h, 5, st);
    return NECG_OK;
}

// Capture the fused launch sequence on the handle's own stream and keep it as
// the handle's graph for `key`.  On any failure the handle keeps no graph for
// the key and the caller launches eagerly.
void capture_fused(necg_handle *h, LaunchArgs &a, double *f_dev, double *g_dev, size_t siv,
                   const necg_handle::GraphKey &key) {
    if (!h->gstream && cudaStreamCreateWithFlags(&h->gstream, cudaStreamNonBlocking) != cudaSuccess) {
        h->gstream = nullptr;
        cudaGetLastError();
        return;
    }
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(h->gstream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    const int rc = enqueue_fused(h, a, f_dev, g_dev, siv, h->gstream);
    const cudaError_t e = cudaStreamEndCapture(h->gstream, &graph);
    cudaGraphExec_t exec = nullptr;
    const bool ok = rc == NECG_OK && e == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    if (!ok) return;
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    h->gexec = exec;
    h->gkey = key;
}

}  // namespace

extern "C" {

int necg_create(int n, int nst, int K_max, double efs, const double *mass_host,
                const double *ncv_host, const double *scvv_host, const double *sml_host,
                const double *sms_host, necg_handle **out) {
    if (!out) return NECG_ERR_ARG;
    *out = nullptr;
    if (n < 1 || n > 6) return NECG_ERR_UNSUPPORTED;
    if (nst < 1 || K_max < 1 || !mass_host || !ncv_host || !scvv_host || !sml_host || !sms_host)
        return NECG_ERR_ARG;
    necg_handle *h = new necg_handle();
    h->n = n;
    h->nst = nst;
    h->K_max = K_max;
    h->efs = efs;
    h->mass.assign(mass_host, mass_host + n * n);
    h->ncv.assign(ncv_host, ncv_host + n + 1);
    h->scvv.assign(scvv_host, scvv_host + nst);
    h->sml.assign(sml_host, sml_host + (size_t)nst * n * n);
    h->sms.assign(sms_host, sms_host + (size_t)nst * 9 * n * n);
    h->sms_general = false;
    for (int p = 0; p < nst && !h->sms_general; ++p)
        for (int r = 0; r < 3 * n && !h->sms_general; ++r)
            for (int c = 0; c < 3 * n && !h->sms_general; ++c) {
                const double *S = &h->sms[(size_t)p * 9 * n * n];
                h->sms_general = S[r * 3 * n + c] != (r % 3 == c % 3 ? S[(r / 3 * 3) * 3 * n + c / 3 * 3] : 0.0);
            }
    // default tile widths per particle count
    h->lc_e = n >= 5 ? 4 : 8;
    h->lc_g = n >= 5 ? 4 : 8;
    cudaGetDevice(&h->device);
    const size_t K = (size_t)K_max;
    const size_t blk = (size_t)(n * (n + 1) / 2 + 3 * n);
    int rc = NECG_OK;
    if (!rc) rc = dalloc(h, &h->d_sml, h->sml.size());
    if (!rc) rc = dalloc(h, &h->d_sms, h->sms.size());
    if (!rc) rc = dalloc(h, &h->d_scvv, (size_t)nst);
    if (!rc) rc = dalloc(h, &h->d_bra, (size_t)necg::bra_record_size(n) * ((K + 31) / 32 * 32));
    if (!rc) rc = dalloc(h, &h->d_ket, (size_t)necg::ket_record_size(n) * K * nst);
    if (!rc) rc = dalloc(h, &h->d_part, necg::part_doubles(n, K_max));
    if (!rc) rc = dalloc(h, &h->d_H, K * K);
    if (!rc) rc = dalloc(h, &h->d_S, K * K);
    if (!rc) rc = dalloc(h, &h->d_rows, 2 * K);
    if (!rc) rc = dalloc(h, &h->d_scal, (size_t)4);
    if (!rc) rc = dalloc(h, &h->d_x, K * blk + K);
    // f, the status words and g side by side, for one copy to the host
    if (!rc) rc = dalloc(h, &h->d_out, kOutHead + K * blk + K);
    if (!rc) {
        h->d_f = h->d_out;
        h->d_status = (int *)(h->d_out + 1);
        h->d_g = h->d_out + kOutHead;
    }
    cudaStream_t ls = rc ? nullptr : lib_stream(h);
    if (!rc) rc = cuda_fail(cudaMemcpyAsync(h->d_sml, h->sml.data(), h->sml.size() * 8, cudaMemcpyHostToDevice, ls));
    if (!rc) rc = cuda_fail(cudaMemcpyAsync(h->d_sms, h->sms.data(), h->sms.size() * 8, cudaMemcpyHostToDevice, ls));
    if (!rc) rc = cuda_fail(cudaMemcpyAsync(h->d_scvv, h->scvv.data(), h->scvv.size() * 8, cudaMemcpyHostToDevice, ls));
    if (!rc) rc = cuda_fail(cudaMemsetAsync(h->d_status, 0, 16, ls));
    if (!rc) rc = setup_symmetric(h);
    // the workspace is allocated in the library stream's order: make it usable on every stream
    if (!rc) rc = cuda_fail(cudaStreamSynchronize(ls));
    if (rc) {
        free_all(h);
        delete h;
        return rc;
    }
    *out = h;
    return NECG_OK;
}

int necg_destroy(necg_handle *h) {
    if (!h) return NECG_ERR_ARG;
    cudaSetDevice(h->device);
    free_all(h);
    if (h->h_out) cudaFreeHost(h->h_out);
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    if (h->gstream) cudaStreamDestroy(h->gstream);
    delete h;
    return NECG_OK;
}

long long necg_workspace_bytes(const necg_handle *h) { return h ? h->ws_bytes : -1; }

int necg_set_tiles(necg_handle *h, int lc_energy, int lc_grad) {
    if (!h || lc_energy < 1 || lc_grad < 4 || lc_energy > 4096 || lc_grad > 4096)
        return NECG_ERR_ARG;
    h->lc_e = lc_energy;
    h->lc_g = lc_grad;
    ++h->gversion;
    return NECG_OK;
}

int necg_set_symmetric(necg_handle *h, int mode, int lc, int minw) {
    const bool blockv = minw == 208 || minw == 216 || minw == 218 || minw == 228 || minw == 222 || minw == 232 || minw == 248 ||
                        minw == 258 || minw == 268;
    const bool okw = minw == 8 || minw == 12 || minw == 16 ||
                     (mode == 2 && (minw == 108 || minw == 112 || minw == 118 || minw == 122 || blockv));
    if (!h || mode < 0 || mode > 2 || lc < 1 || lc > 64 || !okw) return NECG_ERR_ARG;
    if (blockv && !necg::fused_variant_ok(h->n, minw)) return NECG_ERR_UNSUPPORTED;  // shared memory
    if (mode && !h->sym_ok) return NECG_ERR_UNSUPPORTED;
    h->refit = h->refit || h->grad_mode != mode || h->lc_s != lc || h->minb_s != minw;
    h->grad_mode = mode;
    h->lc_s = lc;
    h->minb_s = minw;
    ++h->gversion;
    return NECG_OK;
}

int necg_set_splits(necg_handle *h, int npc) {
    if (!h || npc < 1 || npc > h->nst) return NECG_ERR_ARG;
    h->refit = h->refit || h->npc != npc;
    h->npc = npc;
    ++h->gversion;
    return NECG_OK;
}

int necg_set_variant(necg_handle *h, int minw_energy, int minw_grad) {
    auto okw = [](int w) { return w == 8 || w == 12 || w == 16 || w == 20; };
    if (!h || !okw(minw_energy) || !(okw(minw_grad) || minw_grad == 112 || minw_grad == 116))
        return NECG_ERR_ARG;
    h->minb_e = minw_energy;
    h->minb_g = minw_grad;
    ++h->gversion;
    return NECG_OK;
}

int necg_build_matrices(necg_handle *h, int K, const double *iv_dev, const double *C_dev,
                        double *H_dev, double *S_dev, double *Kin_dev, double *Pot_dev,
                        double *en_dev, void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    if ((rc = ensure_tiles(h, K, st))) return rc;
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = C_dev;
    a.H = H_dev ? H_dev : h->d_H;
    a.S = S_dev ? S_dev : h->d_S;
    a.Kin = Kin_dev;
    a.Pot = Pot_dev;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    necg::launch_energy(a, st);
    if (C_dev && en_dev) necg::launch_rows_finalize(a, nullptr, nullptr, 0, 0.0, 0.0, st, nullptr, en_dev);
    return finish_launch();
}

int necg_outprod(necg_handle *h, int K, const double *x_dev, double *f_dev, double *g_dev,
                 double *H_dev, double *S_dev, void *stream) {
    necg::TraceRange trace("necg_outprod");
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!x_dev || !g_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const bool fused = h->grad_mode == 2;
    if (fused) {  // the status reset is part of the fused launch sequence
        CK(cudaSetDevice(h->device));
        h->last_stream = st;
    } else if ((rc = begin(h, st))) {
        return rc;
    }
    // in fused mode too, which does not read them: a later call that does may be captured
    if ((rc = ensure_tiles(h, K, st))) return rc;
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    LaunchArgs a = base_args(h, K);
    a.iv = x_dev;
    a.C = x_dev + siv;
    a.H = H_dev ? H_dev : h->d_H;
    a.S = S_dev ? S_dev : h->d_S;
    a.g = g_dev;
    int npc = necg::fused_splits(h);
    if (h->grad_mode >= 1 && (rc = ensure_sym_tiles(h, K, st, npc))) return rc;
    if (fused) {
        // fused: one pass over unordered pairs: row sums, both gradients' raw sums of H
        // and of S and, on request, H and S
        sym_args(h, a);
        // H and S are written only for a caller that wants one of them
        if (!H_dev && !S_dev) a.H = a.S = nullptr;
        else if (npc > 1 && (size_t)npc * K * K > h->hp_cap && capturing(st)) npc = 1;  // no buffers for split H and S
        else if ((rc = ensure_split_matrices(h, K, npc, st))) return rc;
        a.npc = npc;
        a.Hp = h->d_Hp;
        a.Sp = h->d_Sp;
        // A call that repeats the previous call's buffers, K and settings
        // replays the captured launch sequence (captured the second time the
        // same key is seen, so callers whose buffers change every call stay
        // eager); a stream that is itself being captured gets the launches.
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CK(cudaStreamIsCapturing(st, &cap));
        const necg_handle::GraphKey key{K, x_dev, f_dev, g_dev, a.H, a.S, h->gversion};
        if (cap == cudaStreamCaptureStatusNone) {
            if (!(h->gexec && h->gkey == key) && h->gseen == key) capture_fused(h, a, f_dev, g_dev, siv, key);
            if (h->gexec && h->gkey == key) {
                CK(cudaGraphLaunch(h->gexec, st));
                return finish_launch();
            }
        }
        h->gseen = key;
        if ((rc = enqueue_fused(h, a, f_dev, g_dev, siv, st))) return rc;
        return finish_launch();
    }
    mark(h, 0, st);
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    mark(h, 1, st);
    necg::launch_energy(a, st);
    mark(h, 2, st);
    necg::launch_rows_finalize(a, f_dev, g_dev + siv, 0, 0.0, 0.0, st);
    if ((rc = launch_gradient(h, a, st))) return rc;
    return finish_launch();
}

// ---- one evaluation split across ranks (tiles of the fused pass) -----------
namespace {
int shard_args(necg_handle *h, int K, const double *x_dev, int t0, int t1, cudaStream_t st, LaunchArgs &a) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!x_dev) return NECG_ERR_ARG;
    if (!h->sym_ok) return NECG_ERR_UNSUPPORTED;
    CK(cudaSetDevice(h->device));
    if ((rc = ensure_sym_tiles(h, K, st, 1))) return rc;
    if (t0 < 0 || t1 < t0 || t1 > h->nstiles) return NECG_ERR_ARG;
    a = base_args(h, K);
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    a.iv = x_dev;
    a.C = x_dev + siv;
    sym_args(h, a);
    a.st_begin = t0;
    a.st_end = t1;
    return NECG_OK;
}
// The per-basis sums of this shard's tiles (all 0 for an empty range, which
// st_end = 0 cannot say).
int shard_sums(const LaunchArgs &a, cudaStream_t st) {
    if (a.st_end > a.st_begin) return necg::launch_fsym_sum(a, st);
    return cudaMemsetAsync(a.part, 0, sizeof(double) * necg::sums_doubles(a.n, a.K), st) == cudaSuccess ? 0 : -1;
}
}  // namespace

int necg_shard_tiles(necg_handle *h, int K, int *ntiles) {
    if (!ntiles) return NECG_ERR_ARG;
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!h->sym_ok) return NECG_ERR_UNSUPPORTED;
    // builds the lists and buffers now, for callers that keep that out of their first
    // step, on whatever stream that will be
    CK(cudaSetDevice(h->device));
    if ((rc = ensure_tiles(h, K, h->last_stream))) return rc;
    if ((rc = ensure_sym_tiles(h, K, h->last_stream, necg::fused_splits(h)))) return rc;
    CK(cudaStreamSynchronize(h->last_stream));
    *ntiles = h->nstiles;
    return NECG_OK;
}

int necg_shard_pairs(necg_handle *h, int K, const double *x_dev, int tile_begin, int tile_end,
                     double *rows_dev, void *stream) {
    necg::TraceRange trace("necg_shard_pairs");
    cudaStream_t st = (cudaStream_t)stream;
    LaunchArgs a;
    int rc = shard_args(h, K, x_dev, tile_begin, tile_end, st, a);
    if (rc) return rc;
    if (!rows_dev) return NECG_ERR_ARG;
    if ((rc = begin(h, st))) return rc;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    if (tile_end > tile_begin && necg::launch_fsym(a, st)) return NECG_ERR_ARG;
    if (shard_sums(a, st)) return NECG_ERR_ARG;
    if (necg::launch_rows_from_sums(a, rows_dev, st)) return NECG_ERR_ARG;
    return finish_launch();
}

int necg_shard_grad(necg_handle *h, int K, const double *x_dev, const double *rows_dev, int tile_begin,
                    int tile_end, double *f_dev, double *g_dev, double *sums_dev, void *stream) {
    necg::TraceRange trace("necg_shard_grad");
    cudaStream_t st = (cudaStream_t)stream;
    LaunchArgs a;
    int rc = shard_args(h, K, x_dev, tile_begin, tile_end, st, a);
    if (rc) return rc;
    if (!rows_dev || !g_dev || !sums_dev) return NECG_ERR_ARG;
    h->last_stream = st;
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    a.g = g_dev;
    a.sums = sums_dev;
    necg::launch_finalize(a, rows_dev, f_dev, g_dev + siv, st);
    if (shard_sums(a, st)) return NECG_ERR_ARG;  // per-basis sums of this shard's tiles only
    if (necg::launch_fsym_finish(a, nullptr, nullptr, false, st)) return NECG_ERR_ARG;
    return finish_launch();
}

int necg_shard_finish(necg_handle *h, int K, const double *x_dev, const double *sums_dev, double *g_dev,
                      void *stream) {
    necg::TraceRange trace("necg_shard_finish");
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!x_dev || !sums_dev || !g_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(h->device));
    h->last_stream = st;
    LaunchArgs a = base_args(h, K);
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    a.iv = x_dev;
    a.C = x_dev + siv;
    a.g = g_dev;
    if (necg::launch_reduce_sums(a, sums_dev, st)) return NECG_ERR_ARG;
    return finish_launch();
}

int necg_outprod_host(necg_handle *h, int K, const double *x_host, double *f_host,
                      double *g_host, void *stream) {
    necg::TraceRange trace("necg_outprod_host");
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!x_host || !g_host) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(h->device));
    const size_t len = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n) + K;
    CK(cudaMemcpyAsync(h->d_x, x_host, len * sizeof(double), cudaMemcpyHostToDevice, st));
    rc = necg_outprod(h, K, h->d_x, h->d_f, h->d_g, nullptr, nullptr, stream);
    if (rc) return rc;
    // f, the status words and g come back in one copy into a pinned buffer of the
    // handle, and the stream is waited for once; a g_host that is not ordinary
    // memory of the process (pinned, managed, or a device address, for which the
    // runtime decides) gets its copy straight, since a copy into pageable memory
    // would go through the driver's own staging, one more wait
    if (!h->h_out) CK(cudaMallocHost((void **)&h->h_out, (kOutHead + (size_t)h->K_max * (len / K)) * sizeof(double)));
    cudaPointerAttributes at;
    const cudaError_t known = cudaPointerGetAttributes(&at, g_host);
    if (known != cudaSuccess) cudaGetLastError();
    const bool direct = known == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    CK(cudaMemcpyAsync(h->h_out, h->d_out, (kOutHead + (direct ? 0 : len)) * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (direct) CK(cudaMemcpyAsync(g_host, h->d_g, len * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (!direct) memcpy(g_host, h->h_out + kOutHead, len * sizeof(double));
    if (f_host) *f_host = h->h_out[0];
    int sw[2];
    memcpy(sw, h->h_out + 1, sizeof(sw));
    return status_code(sw, nullptr);
}

int necg_make_grad(necg_handle *h, int K, const double *iv_dev, const double *C_dev,
                   const double *H_dev, const double *S_dev, double eng, double norm,
                   double *g_dev, void *stream) {
    necg::TraceRange trace("necg_make_grad");
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || !C_dev || !H_dev || !S_dev || !g_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = C_dev;
    a.H = const_cast<double *>(H_dev);
    a.S = const_cast<double *>(S_dev);
    a.g = g_dev;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    // GRADC = 2 norm (H - eng S) C with the caller's eng and norm; also sets
    // the E and norm the gradient tiles read
    necg::launch_rows_finalize(a, nullptr, g_dev + siv, 1, eng, norm, st);
    if ((rc = launch_gradient(h, a, st))) return rc;
    return finish_launch();
}

int necg_make_grad_dev(necg_handle *h, int K, const double *iv_dev, const double *C_dev,
                       const double *H_dev, const double *S_dev, const double *en_dev, double *g_dev,
                       void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || !C_dev || !H_dev || !S_dev || !en_dev || !g_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    const size_t siv = (size_t)K * (h->n * (h->n + 1) / 2 + 3 * h->n);
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = C_dev;
    a.H = const_cast<double *>(H_dev);
    a.S = const_cast<double *>(S_dev);
    a.g = g_dev;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    necg::launch_rows_finalize(a, nullptr, g_dev + siv, 2, 0.0, 0.0, st, en_dev, nullptr);
    if ((rc = launch_gradient(h, a, st))) return rc;
    return finish_launch();
}

int necg_matel(necg_handle *h, int K, const double *iv_dev, int nterms, const int *terms_dev,
               double *out_dev, void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || nterms < 0 || (nterms > 0 && (!terms_dev || !out_dev))) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = nullptr;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    if (nterms > 0) necg::launch_matel(a, terms_dev, nterms, out_dev, st);
    return finish_launch();
}

int necg_rrms(necg_handle *h, int K, const double *iv_dev, int nterms, const int *terms_dev,
              double *out_dev, void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || nterms < 0 || (nterms > 0 && (!terms_dev || !out_dev))) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = nullptr;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    if (nterms > 0) necg::launch_rrms(a, terms_dev, nterms, out_dev, st);
    return finish_launch();
}

int necg_dipole(necg_handle *h, int K, const double *iv_dev, const double *C_dev, double *comps_dev,
                double *dipole_dev, void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || !C_dev || !comps_dev) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    if ((rc = ensure_tiles(h, K, st))) return rc;
    if ((rc = setup_dipole(h, st))) return rc;
    LaunchArgs a = base_args(h, K);
    // the tile partials reuse the gradient-partial workspace
    const size_t need = (size_t)a.ntiles * (3 * h->n + 1);
    const size_t cap = necg::part_doubles(h->n, h->K_max);
    if (need > cap) return NECG_ERR_CAPACITY;
    a.iv = iv_dev;
    a.C = C_dev;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    necg::launch_dipole(a, h->d_part, cap, comps_dev, dipole_dev, st);
    return finish_launch();
}

int necg_gradel(necg_handle *h, int K, const double *iv_dev, int nterms, const int *terms_dev,
                double *tgvl_dev, double *tgvls_dev, void *stream) {
    int rc = check_K(h, K);
    if (rc) return rc;
    if (!iv_dev || nterms < 0 || (nterms > 0 && (!terms_dev || !tgvl_dev || !tgvls_dev)))
        return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = begin(h, st))) return rc;
    LaunchArgs a = base_args(h, K);
    a.iv = iv_dev;
    a.C = nullptr;
    if (necg::launch_prep(a, st)) return NECG_ERR_UNSUPPORTED;
    if (nterms > 0) necg::launch_gradel(a, terms_dev, nterms, tgvl_dev, tgvls_dev, st);
    return finish_launch();
}

int necg_f0(const double *z_dev, int count, double *f_dev, double *df_dev, void *stream) {
    if (count < 0 || (count > 0 && !z_dev)) return NECG_ERR_ARG;
    if (count == 0) return NECG_OK;
    necg::launch_f0(z_dev, count, f_dev, df_dev, (cudaStream_t)stream);
    return finish_launch();
}

int necg_status(necg_handle *h, long long *bad_pair) {
    if (!h) return NECG_ERR_ARG;
    CK(cudaSetDevice(h->device));
    int st[2];
    CK(cudaMemcpyAsync(st, h->d_status, sizeof(st), cudaMemcpyDeviceToHost, h->last_stream));
    CK(cudaStreamSynchronize(h->last_stream));
    return status_code(st, bad_pair);
}

int necg_profile(necg_handle *h, int enable) {
    if (!h) return NECG_ERR_ARG;
    CK(cudaSetDevice(h->device));
    if (enable && !h->ev[0])
        for (cudaEvent_t &e : h->ev) CK(cudaEventCreate(&e));
    h->profile = enable != 0;
    ++h->gversion;
    return NECG_OK;
}

int necg_phase_ms(necg_handle *h, double *ms) {
    if (!h || !ms || !h->ev[0]) return NECG_ERR_ARG;
    CK(cudaSetDevice(h->device));
    CK(cudaEventSynchronize(h->ev[5]));
    for (int i = 0; i < 5; ++i) {
        float t = 0.f;
        CK(cudaEventElapsedTime(&t, h->ev[i], h->ev[i + 1]));
        ms[i] = t;
    }
    return NECG_OK;
}

int necg_fp64_peak(int iters, double *tflops, void *stream) {
    if (iters < 1 || !tflops) return NECG_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = sms * 8;
    double *sink = nullptr;
    CK(cudaMalloc((void **)&sink, blocks * sizeof(double)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    necg::launch_fp64_probe(blocks, iters / 4 + 1, sink, st);  // warm-up
    cudaEventRecord(e0, st);
    necg::launch_fp64_probe(blocks, iters, sink, st);
    cudaEventRecord(e1, st);
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (e != cudaSuccess) return cuda_fail(e);
    const double flops = 2.0 * 8.0 * (double)iters * blocks * 256.0;
    *tflops = flops / (ms * 1e-3) / 1e12;
    return NECG_OK;
}

const char *necg_status_string(int code) {
    switch (code) {
    case NECG_OK: return "ok";
    case NECG_ERR_ARG: return "invalid argument";
    case NECG_ERR_NOT_PD: return "A_k + A_l' is not positive definite for some basis pair";
    case NECG_ERR_NONFINITE: return "non-finite energy or gradient";
    case NECG_ERR_CUDA: return "CUDA runtime error";
    case NECG_ERR_ALLOC: return "device allocation failed";
    case NECG_ERR_UNSUPPORTED: return "unsupported particle count (1..6)";
    case NECG_ERR_CAPACITY: return "K exceeds the handle's K_max";
    default: return "unknown status";
    }
}

}  // extern "C"
