// necg_handle.h -- internal layout of the opaque necg_handle (one particle
// system + symmetry set + device workspace for bases of up to K_max functions).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "necg_tiles.h"
#include "../../include/necg.h"

struct necg_handle {
    int n, nst, K_max;
    double efs;
    std::vector<double> mass, ncv, scvv, sml, sms;
    double *d_sml = nullptr, *d_sms = nullptr, *d_scvv = nullptr;
    double *d_bra = nullptr, *d_ket = nullptr, *d_part = nullptr;
    double *d_H = nullptr, *d_S = nullptr, *d_rows = nullptr, *d_scal = nullptr;
    double *d_x = nullptr, *d_g = nullptr, *d_f = nullptr;
    int *d_status = nullptr;
    int2 *d_tiles = nullptr;
    size_t tiles_cap = 0;
    int tiles_K = -1, tiles_lc = -1, ntiles = 0;
    int lc_e = 8, lc_g = 8;
    int minb_e = 16, minb_g = 8;
    int device = 0;
    cudaStream_t last_stream = nullptr;
    long long ws_bytes = 0;
    bool profile = false;
    cudaEvent_t ev[6] = {};
    double *d_dipcls = nullptr;  // classes of the dipole's terms (set when the symmetry set is a group)
    bool dip_ready = false;      // ... looked for
    // symmetric gradient pass (when the symmetry set is closed under inverse)
    bool sym_ok = false;
    int grad_mode = 0;  // 0 ordered pairs, 1 symmetric, 2 fused energy + symmetric
    int lc_s = 4, minb_s = 8;
    int *d_pinv = nullptr;
    int *d_kcnt = nullptr, *d_ksrc = nullptr;
    double *d_kcoef = nullptr;
    int kmaxnz = 0, kfold = 0;  // the ket frame map (RawMap)
    // tile lists of the symmetric passes and the queue of the block variants, in one
    // buffer (lists points into it)
    int2 *d_lists = nullptr;
    size_t lists_cap = 0;  // int2
    necg::SymLists lists = {};
    necg::SymQueue queue = {};
    int stiles_K = -1, stiles_lc = -1, nstiles = 0, nbgroups = 0, sgroups_w = 0;
    double *d_psym = nullptr;
    size_t psym_cap = 0;  // doubles
    double *d_xsym = nullptr;  // parts after the first of the queue's split tail groups
    size_t xsym_cap = 0;  // doubles
    bool sms_general = true;   // some shift map is not kron(m, I3)
    int *d_qcount = nullptr;    // queue head of the block-synchronised fused pass
    // fused pass with one-warp tiles: symmetry terms split over npc warps per tile
    int npc = 1;
    bool refit = false;  // the pass's settings changed: its buffers are made to measure with the next lists
    double *d_Hp = nullptr, *d_Sp = nullptr;  // npc K x K sums each, when the caller wants H and S
    size_t hp_cap = 0;                        // doubles per buffer
    double *d_out = nullptr;  // f, the status words and g (d_f, d_status and d_g point into it)
    double *h_out = nullptr;  // its pinned copy, of the host entry point
    // the fused evaluation's launch sequence as a CUDA graph: captured (on the
    // handle's own stream) the second time a call repeats the same key, then
    // replayed on the caller's stream while the key stays the same
    struct GraphKey {
        int K = -1;
        const void *x = nullptr, *f = nullptr, *g = nullptr, *H = nullptr, *S = nullptr;
        int version = -1;
        bool operator==(const GraphKey &o) const {
            return K == o.K && x == o.x && f == o.f && g == o.g && H == o.H && S == o.S && version == o.version;
        }
    };
    int gversion = 0;  // bumped by every change of settings, tiles or buffers
    GraphKey gkey, gseen;
    cudaGraphExec_t gexec = nullptr;
    cudaStream_t gstream = nullptr;
};

namespace necg {
// Tile list and partial buffers of the fused pass for bases of K functions
// (the handle's ket chunk lc_s), as the batched step needs them; returns a
// status code.  May synchronise `st` when the list changes.
int prepare_fused(necg_handle *h, int K, cudaStream_t st);
// Splits of the symmetry terms per one-warp tile of the fused pass (1: none):
// npc when the handle runs the fused pass with a one-warp variant, else 1.
inline int fused_splits(const necg_handle *h) {
    return h->grad_mode == 2 && h->minb_s < 200 && h->npc > 1 ? h->npc : 1;
}
}  // namespace necg
