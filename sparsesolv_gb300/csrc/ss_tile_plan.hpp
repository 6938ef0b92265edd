// ss_tile_plan.hpp -- the tile sweep's schedule, computed on the host from a
// level-ordered triangle (plain C++: the sweep's launcher in ss_tile.cu and a
// CPU test that emulates the schedule both compile it).
//
// A tile is a contiguous range of rows in solve order (ascending rows for a
// lower triangle, descending for an upper one). A triangle's dependencies all
// point to earlier rows, so tiles depend on lower-numbered tiles only, whatever
// the pattern: tile order is a topological order and any dependency path crosses
// each tile border at most once.
//
// Inside a tile the rows are taken level by level in groups of rows of one level,
// one warp a group. Two ways of summing a row:
//   * by age (real values): oldest dependency first, the entries more than TS_TAILS
//     levels up alternately into two partial sums, in columns over one or two lanes
//     a row, each block of four columns waiting for what it reads; then those
//     TS_TAILS, ..., 1 levels up, a stage for each distance, on one lane a row. The
//     values are stored pre-scaled by the row's 1/L_ii or D_i, so the work left when
//     the last dependency arrives is one fused multiply-add an entry, and every
//     earlier entry has as many levels' time as it is levels up;
//   * by lanes (complex values): lane q of `lanes` sums every lanes-th entry from q
//     in column order, a step of one entry a lane waiting for what it reads, then a
//     butterfly: the arithmetic of the cluster and sync-free sweeps, bit for bit.
//     The iterates of the singular complex systems are sensitive to rounding. Two
//     GPU lanes share a lane's sum, one its real and one its imaginary part, which
//     halves the FP64 instructions between a dependency and the row's result.
// Both depend on the row alone and not on how rows fall into tiles and groups.
//
// Values a group reads come from two shared-memory rings: the tile's own values
// by production position, and values of other tiles ("halo") by their place in
// the tile's halo list, ordered by dependency level and delivered in that order.
// An entry whose ring slot would be reused before the read is "far": it is
// read from the output vector in memory, in its place in the sum, where every
// value is its own ready flag. Every wait is for an earlier group, an earlier
// halo value or a lower tile.
//
// CS consecutive tiles run on one thread-block cluster. A halo value of the first lap
// of the ring whose tile runs on the same cluster is not polled for in memory: the
// row's owner stores it into the reader's ring slot, which no one else writes before
// its readers are done.
#pragma once

#include <vector>

#ifdef __CUDACC__
#define SSG_HD __host__ __device__
#else
#define SSG_HD
#endif

namespace ssg {

constexpr int TS_W = 12;                  // compute warps
constexpr int TS_R = 4;                   // receiver warps
constexpr int TS_THREADS = 32 * (TS_W + TS_R + 1);  // and one warp that stages records
constexpr int TS_NM = 60;                 // staged groups at most (one barrier each; a multiple of TS_W)
constexpr int TS_TAILS = 2;               // tail stages
constexpr int TS_TAIL = 6;                // entries a row has in one tail stage at most; the rest go to the columns
constexpr int TS_SMEM_MAX = 220 * 1024;   // dynamic shared memory of a CTA

SSG_HD inline int ts_al16(int x) { return (x + 15) & ~15; }

// Shared-memory carve-up, by value size and way of summing.
struct TileLayout {
    int S_own, S_halo;   // ring slots (powers of two); slot S_own + S_halo holds zero (padding entries)
    int B_rec;           // bytes of the record ring
    int o_x, o_full, o_place, o_prog, o_rec, total;
};
TileLayout tile_layout(int elem, int lanes);

// One group's record, staged with one bulk copy. Lanes of a row are r * G .. r * G + G - 1 in the columns, r in the tails
// (by lanes: entry lane l is GPU lanes 2 l and 2 l + 1, and only 16 entry lanes are used);
// every array of values or codes holds all 32 lanes (padding lanes and columns: value 0, the ring slot that holds zero),
// so the kernel's loads have constant strides and no bounds.
//   [0]   16 ints: {cnt | lg G << 8 | K1 << 16 | K2 << 20, blocks | has far entries << 16, first own slot,
//          columns in the first block, per tail stage, oldest first, the last own group it needs (-1: none) and the halo
//          values it needs, KP, o_push / 16, 0, 0,
//          offsets / 16: o_old | o_tail << 16, o_cold | o_ctail << 16, o_cfar, o_row | o_lv << 16}
//   need  per block {last own group needed, halo values needed}; a block is four columns, or one step by lanes
//   rows  cnt row ids
//   lv    cnt values: 1 / L_ii or D_i
//   old   per block its values of every lane (ts_col); tails (K1 + K2) x 32 values
//   codes old (per block those of a lane together) and tails as unsigned shorts: ring slots, TS_FAR for a far entry
//   cfar  with far entries: per old code the row id
//   push  KP x 32 (by row): rank << 20 | ring slot of a CTA of the cluster that reads the row, -1
// By age, a row's entries fill the last columns, so that a block's entries are about equally old in every row; the first
// block's leading columns may be empty in all rows and are skipped.
constexpr int TS_FAR = 0xFFFF;
struct TileRec {
    int o_need, o_row, o_lv, o_old, o_tail, o_cold, o_ctail, o_cfar, o_push, size;
};
SSG_HD inline TileRec tile_rec(int cnt, int nb, int blk, bool far, int KT, int KP, int elem) {
    TileRec r;
    r.o_need = 64;
    r.o_row = r.o_need + ts_al16(8 * nb);
    r.o_lv = r.o_row + ts_al16(4 * cnt);
    r.o_old = r.o_lv + ts_al16(elem * cnt);
    r.o_tail = r.o_old + elem * 32 * blk * nb;
    r.o_cold = r.o_tail + elem * 32 * KT;
    r.o_ctail = r.o_cold + 2 * 32 * blk * nb;
    r.o_cfar = r.o_ctail + 2 * 32 * KT;
    r.o_push = r.o_cfar + (far ? 4 * 32 * blk * nb : 0);
    r.size = r.o_push + 4 * 32 * KP;
    return r;
}
// index of column q of a lane in its block's values: 16 bytes a lane at a time
SSG_HD inline int ts_col(int q, int lane, int blk, int elem) {
    const int vp = blk == 1 ? 1 : 16 / elem;
    return (q / vp) * 32 * vp + lane * vp + q % vp;
}

// tiles: per tile {first group, groups, first halo chunk, halo chunks}
// groups: per group {record offset / 16, record bytes / 16, ring offset / 16, group that must be done before the copy}
// halo: row ids, 32 a chunk (-1: padding, -2: stored into its slot by a tile of the cluster); rel: per 32 of them the group up
// to which all must be done before they are delivered (-1: none)
// dval: per entry of the level-ordered triangle its element index in rec, -1: the diagonal;
// dlv: per level-ordered row the element index of its lv
struct TilePlanHost {
    bool ok = false;
    const char *why = "";
    int T = 0, CS = 1, nfar = 0, npush = 0;
    long long rec_bytes = 0;
    TileLayout lay{};
    std::vector<int> tiles, groups, halo, rel, dval, dlv;
    std::vector<std::vector<unsigned char>> rec;  // per tile, concatenated in order
    std::vector<long long> rec_off;               // per tile, bytes
};

int tile_count(int n, int lanes);
int tile_cluster(int T, int lanes);

// What a plan may cost before the sync-free sweep is the better choice; a plan beyond it is refused.
struct TileLimits {
    double chunks_per_level;  // halo chunks of the tile with most of them, over the triangle's levels
    double far_per_row;       // far entries, over the rows
    long long bytes;          // of the records
};
TileLimits tile_limits(int lanes, long long device_bytes);
// n rows: prp/pci the level-ordered rows (columns as row ids, the diagonal included), ipos[row] position of a row,
// level[row]; lower: solve order is ascending rows. lanes: 0 sums by age, 4 or 8 by lanes. T tiles (<= 0: tile_count), CS
// of them a cluster. lim: null for a plan at any cost.
TilePlanHost tile_plan_host(int n, int nlev, const int *prp, const int *pci, const int *ipos, const int *level,
                            bool lower, int elem, int lanes, int T, int CS, const TileLayout *lay = nullptr,
                            const TileLimits *lim = nullptr);

}  // namespace ssg
