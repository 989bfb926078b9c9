// necg_tiles.h -- the tile lists of the pair passes, in closed form: counts for the
// host, entries for the kernel that fills the lists on the device (and for the
// host emulation).  Nothing is built on the host or copied: filling the lists of
// K = 2048 on the CPU and copying them from pageable memory took up to 0.5 ms of an
// engine's first evaluation.
#pragma once
#include "necg_math.cuh"

namespace necg {

// Tiles of row block kb: ket chunks of LC up to the block's last row.
NECG_HD int block_tiles(int K, int LC, int kb) { return row_last(K, kb) / LC + 1; }
// Tiles of the row blocks before kb (kb = row_blocks(K): all).
NECG_HD int tiles_before(int K, int LC, int kb) {
    int n = 0;
    for (int b = 0; b < kb; ++b) n += block_tiles(K, LC, b);
    return n;
}
// Groups of w consecutive tiles of one row block, the blocks in decreasing order
// (the largest first): those of the blocks after kb (kb = -1: all).
NECG_HD int groups_before(int K, int LC, int w, int kb) {
    int n = 0;
    for (int b = row_blocks(K) - 1; b > kb; --b) n += (block_tiles(K, LC, b) + w - 1) / w;
    return n;
}

// Warps per energy tile: one, or for bases with few tiles up to 8 that share a tile's
// symmetry terms, until there are 12 per SM (matrices of LiH K = 301 on a B200, chunk
// 2: 170 us with 8 per SM, 158 with 12, 157 with 16).
NECG_HD int energy_warps(int nst, int ntiles, int sms) {
    int w = 1;
    while (2 * w <= nst && w < 8 && ntiles * w < 12 * sms) w *= 2;
    return w;
}

// A tile group of the block variants: row block kb, first ket chunk lc0 and, for
// a split group of the queue's tail, its part and the number of parts (one part
// per range of symmetry terms).
__host__ __device__ inline int2 sgroup_pack(int kb, int lc0, int part, int parts) {
    return make_int2(kb, lc0 | part << 24 | (parts - 1) << 28);
}
__host__ __device__ inline int sgroup_lc0(int2 g) { return g.y & 0xffffff; }
__host__ __device__ inline int sgroup_part(int2 g) { return (g.y >> 24) & 0xf; }
__host__ __device__ inline int sgroup_parts(int2 g) { return ((g.y >> 28) & 0x7) + 1; }

// The queue of the block variants: G groups of w tiles.  They are equal work and
// one block per SM takes them, so the last round would run G mod SMs groups while
// the other SMs idle: each of those T groups is split into `parts` units over the
// symmetry terms (as many as keep the round within one unit per SM, at most 8;
// the kernel gives the parts balanced ranges of terms).  Bra partials are
// written per unit into the slots sized for the tiles, so the units must not
// outnumber the tiles.
struct SymQueue {
    int K, LC, w, ntiles, G, tail0, ntail, parts;
    NECG_HD int unit(int group) const { return group < tail0 ? group : tail0 + (group - tail0) * parts; }
    NECG_HD int units() const { return unit(G); }
};
NECG_HD SymQueue sym_queue(int K, int LC, int w, int nst, int sms) {
    SymQueue q{K, LC, w, tiles_before(K, LC, row_blocks(K)), groups_before(K, LC, w, -1), 0, 0, 1};
    const int T = q.G % sms;
    int parts = T > 0 ? sms / T : 1;
    if (parts > 8) parts = 8;
    if (parts > nst) parts = nst;
    if (T > 0 && parts > 1 + (q.ntiles - q.G) / T) parts = 1 + (q.ntiles - q.G) / T;
    q.tail0 = q.G;
    if (parts >= 2) {
        q.tail0 = q.G - T;
        q.ntail = T;
        q.parts = parts;
    }
    return q;
}

// Where the lists go (bgroups, burange: groups of 8 without a split tail, for the
// batched step).
struct SymLists {
    int2 *tiles;           // (kb, lc)
    int *start;            // first tile of each row block (row_blocks + 1)
    int2 *groups;          // the queue's units
    int2 *urange;          // units of each row block
    int *tslot;            // first slot in xsym of each tile of a split group, else -1
    int2 *bgroups, *burange;
};

// Row block kb's entries; thread j of nj.
NECG_HD void fill_sym_lists(const SymQueue &q, const SymLists &o, int kb, int j, int nj) {
    const int nt = block_tiles(q.K, q.LC, kb), t0 = tiles_before(q.K, q.LC, kb);
    const int g0 = groups_before(q.K, q.LC, q.w, kb), ng = (nt + q.w - 1) / q.w;
    const int b0 = groups_before(q.K, q.LC, 8, kb), nb = (nt + 7) / 8;
    if (j == 0) {
        o.start[kb] = t0;
        if (kb == row_blocks(q.K) - 1) o.start[kb + 1] = t0 + nt;
        o.urange[kb] = make_int2(q.unit(g0), q.unit(g0 + ng));
        o.burange[kb] = make_int2(b0, b0 + nb);
    }
    for (int lc = j; lc < nt; lc += nj) {
        o.tiles[t0 + lc] = make_int2(kb, lc);
        const int g = g0 + lc / q.w;
        o.tslot[t0 + lc] = g < q.tail0 ? -1 : ((g - q.tail0) * q.w + lc % q.w) * (q.parts - 1);
    }
    for (int i = j; i < ng; i += nj) {
        const int g = g0 + i, parts = g < q.tail0 ? 1 : q.parts;
        for (int p = 0; p < parts; ++p) o.groups[q.unit(g) + p] = sgroup_pack(kb, i * q.w, p, parts);
    }
    for (int i = j; i < nb; i += nj) o.bgroups[b0 + i] = make_int2(kb, 8 * i);
}

}  // namespace necg
