// ss_tile_plan.cpp -- the tile sweep's schedule (ss_tile_plan.hpp says what it is, ss_tile.cu runs it).
//
// Tiles are planned independently of each other, on host threads; the outputs are put in tile order, so the plan does
// not depend on the thread count (SSG_PLAN_THREADS, 1-64).
#include "ss_tile_plan.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <exception>
#include <memory>
#include <thread>

namespace ssg {

TileLayout tile_layout(int elem, int lanes) {
    TileLayout L{};
    // By age 16 KB for the own ring and 64 KB for the halo ring, whose first lap the cluster's other tiles store into: a tile
    // reads about twice as many rows of other tiles as it has. Measured, us a forward sweep at 41^3 and 80^3 with 32 + 32 KB
    // 347, 1,050; 32 + 64 326, 949; 16 + 64 324, 927; 16 + 128 (too little is left for records) 350, 884. By lanes 32 KB each
    // (16 + 64 KB: 33^3 640 -> 664). The rest stages records.
    L.S_own = (lanes ? 32 : 16) * 1024 / elem;
    L.S_halo = (lanes ? 32 : 64) * 1024 / elem;
    int o = 0;
    L.o_x = o;
    o += ts_al16((L.S_own + L.S_halo + 1) * elem);
    L.o_full = o;
    o += 8 * TS_NM;
    L.o_place = o;
    o += 4 * TS_NM;
    L.o_prog = o;  // compute warps' next groups, then the number of halo values delivered
    o += 4 * 32;
    L.o_rec = o;
    // the kernel loads two tail entries of a stage ahead, whether or not it has them
    const int slack = 64 * elem + 128;
    L.B_rec = (TS_SMEM_MAX - o - slack) & ~15;
    L.total = o + L.B_rec + slack;
    return L;
}

// More tiles put fewer rows of a level on an SM, each border costs its latency once. Measured (us a forward sweep by age, in
// clusters from 8 tiles on): 2,430 rows 1 tile 55, 3 tiles 54; 21,660 rows 8 tiles 125, 12 120, 15 120; 48,800 rows 16 168,
// 24 159; 83,700 rows 20 227, 32 204, 40 207; 196,800 rows 36 338, 50 311, 71 321; 405,000 rows 72 494, 104 454, 128 457;
// 626,580 rows 120 616, 160 565, 200 564; 1,497,840 rows 250 992, 304 927, 380 911, 400 911. 0.0044 n^0.8 is 2, 13, 25, 38, 75,
// 135, 191 and 383. Groups by lanes hold few rows, and want more tiles, most so where there are few of them: complex 101,376
// rows 44 tiles 820, 110 643, 152 622; 626,580 rows 155 tiles 1,947, 300 1,432, 400 1,310; 0.035 n^0.7 is 112 and 400.
int tile_count(int n, int lanes) {
    const int t = (int)std::lround(lanes ? 0.035 * std::pow((double)n, 0.7) : 0.0044 * std::pow((double)n, 0.8));
    return std::max(1, std::min(t, n));
}

// Tiles of a cluster. The next tiles wait for all of a cluster's, so clusters pay where most tiles run at once and a level
// is one group's work, and cost where the GPU's tiles at a time set the pace: by lanes, with 2 to 4 rows a group, 60^3 took
// 1,360 us with 1, 1,437 with 4 and 1,593 with 8 (33^3 664, 655, 651). By age, 1 against 8: 3 tiles 54 / 57, 20^3 123 / 120,
// 41^3 384 / 324, 80^3 1,101 / 927; 16 gives 80^3 918 and 41^3 311 instead of 316 (50 tiles): not worth the larger clusters,
// of which fewer fit beside other work.
int tile_cluster(int T, int lanes) { return lanes || T < 8 ? 1 : 8; }

// Consecutive rows make good tiles where a row's dependencies are near it in the order: a breadth-first or banded order, a
// grid's natural one. In an order that scatters them a tile reads rows of most lower tiles, 32 (a chunk) at a time in level
// order at about 0.4 us by age and 1 us by lanes, and a triangle of few levels is soon through without tiles: the sync-free
// sweep takes about 1.3 us a level (complex 2). Measured, us a sweep forward, tiles / sync-free, by halo chunks a level of the
// tile with most. By age, rows in random order: curl-curl 10^3 0.8 34 / 68, 12^3 1.7 47 / 78, 14^3 3.1 61 / 77, 16^3 4.8
// 111 / 82, 20^3 8.8 226 / 84, 24^3 14 324 / 86; 27-point 16^3 2.1 40 / 61, 28^3 11 172 / 71; 7-point 16^3 5.6 29 / 26, 40^3 18
// 95 / 35. (Breadth-first curl-curl orders have 0.2, natural grids up to 0.6.) By lanes: 9^3 0.9 88 / 108, 10^3 1.3 104 / 110,
// 11^3 1.6 133 / 117, 16^3 3.9 254 / 136, 24^3 7.7 459 / 147. Far entries are polled in memory one by one on a row's chain:
// orders shuffled within a window have few chunks and many of them. Far entries a row, us tiles / sync-free, complex 24^3 with
// windows of 500, 2,000 and 6,000 rows: 0.04 1,459 / 1,712, 0.6 1,653 / 1,306, 3.7 1,574 / 734; real 40^3: 0.01 896 / 1,986,
// 0.08 1,537 / 1,739, 0.07 1,713 / 1,328.
// Memory. A record holds 32 lanes whatever its group has, so its bytes over the triangle's CSR bytes are about 2 where levels
// are wide (breadth-first curl-curl 80^3 1.9, 27-point 80^3 1.6, complex 4 to 5), and up to 20 where a level is one row
// (tridiagonal 17, bands 14 to 16); the tiles are 3 to 4 times faster there all the same (band of 16, 50,000 rows: 12 against
// 46 ms). The records, which the host holds too while it plans, may take a sixteenth of the device's memory (17 GB).
TileLimits tile_limits(int lanes, long long device_bytes) { return {lanes ? 1.0 : 3.0, 0.1, device_bytes / 16}; }

namespace {

struct TileOut {
    std::vector<int> groups, halo, rel;  // ring offsets and groups relative to the tile
    std::vector<unsigned char> rec;
    int nfar = 0;
    const char *why = nullptr;
};

struct Ctx {
    int n, elem, lanes;
    const int *prp, *pci, *ipos, *level;
    bool lower;
    TileLayout L;
    int *dval, *dlv;  // element indices relative to the tile's records; made absolute afterwards
    int row(int p) const { return lower ? p : n - 1 - p; }
    int ord(int i) const { return lower ? i : n - 1 - i; }
};

struct Entry {
    int lev, j, k;   // dependency level, row, index in the level-ordered triangle
};

// scratch of one planning thread
struct Scratch {
    std::vector<int> hpos;  // row -> halo position of the current tile, -1
    explicit Scratch(int n) : hpos((size_t)n, -1) {}
};

// the rows of other tiles that a tile reads, in (level, order), and which of them are pushed to it
struct Halo {
    std::vector<int> row;
    std::vector<unsigned char> pushed;
    const char *why = nullptr;
};

void find_halo(const Ctx &C, int p0, int p1, Scratch &S, Halo &H) {
    for (int p = p0; p < p1; ++p) {
        const int i = C.row(p), t = C.ipos[i];
        for (int k = C.prp[t]; k < C.prp[t + 1]; ++k) {
            const int j = C.pci[k];
            if (j == i) continue;
            if (j < 0 || j >= C.n || C.ord(j) >= p || C.level[j] >= C.level[i]) {
                H.why = "an entry is not a dependency of its row";
                break;
            }
            if (C.ord(j) < p0 && S.hpos[j] < 0) {
                S.hpos[j] = 0;
                H.row.push_back(j);
            }
        }
    }
    std::sort(H.row.begin(), H.row.end(), [&](int a, int b) {
        return C.level[a] != C.level[b] ? C.level[a] < C.level[b] : C.ord(a) < C.ord(b);
    });
    H.pushed.assign(H.row.size(), 0);
    for (int h : H.row) S.hpos[h] = -1;
}

// per place of the solve order from p0 on, the ring slots of the cluster's CTAs that take its row: rank << 20 | slot
struct Push {
    int p0 = 0;
    std::vector<int> ptr, dat;
    int count(int p) const { return ptr.empty() ? 0 : ptr[p - p0 + 1] - ptr[p - p0]; }
};

// the first lap's values that tiles t0 to t1 - 1 take from each other
template <typename F>
void find_pushes(const Ctx &C, int t0, int t1, const F &first, std::vector<Halo> &halo, Push &P) {
    P.p0 = first(t0);
    P.ptr.assign((size_t)(first(t1) - P.p0) + 2, 0);
    auto each = [&](auto f) {
        for (int t = t0; t < t1; ++t) {
            const int m = std::min((int)halo[t].row.size(), C.L.S_halo);
            for (int q = 0; q < m; ++q) {
                const int p = C.ord(halo[t].row[q]) - P.p0;
                if (p >= 0) f(t, q, p);
            }
        }
    };
    each([&](int t, int q, int p) {
        halo[t].pushed[q] = 1;
        P.ptr[p + 2]++;
    });
    for (size_t p = 2; p < P.ptr.size(); ++p) P.ptr[p] += P.ptr[p - 1];
    P.dat.resize((size_t)P.ptr.back());
    each([&](int t, int q, int p) { P.dat[P.ptr[p + 1]++] = (t - t0) << 20 | q; });  // leaves ptr[p + 1] at the end of p
}

void plan_tile(const Ctx &C, int p0, int p1, const Halo &halo, const Push &pushes, Scratch &S, TileOut &O) {
    const int nr = p1 - p0, elem = C.elem;
    const TileLayout &L = C.L;
    // rows in (level, order), and groups of rows of one level
    int lmin = 1 << 30, lmax = 0;
    for (int p = p0; p < p1; ++p) {
        const int l = C.level[C.row(p)];
        lmin = std::min(lmin, l);
        lmax = std::max(lmax, l);
    }
    std::vector<int> cnt((size_t)(lmax - lmin) + 2, 0), rows((size_t)nr), pos((size_t)nr), grp((size_t)nr);
    for (int p = p0; p < p1; ++p) cnt[C.level[C.row(p)] - lmin + 1]++;
    for (size_t l = 1; l < cnt.size(); ++l) cnt[l] += cnt[l - 1];
    {
        std::vector<int> at(cnt.begin(), cnt.end() - 1);
        for (int p = p0; p < p1; ++p) {
            const int q = at[C.level[C.row(p)] - lmin]++;
            rows[q] = p;
            pos[p - p0] = q;
        }
    }
    std::vector<int> gfirst;
    const int most = C.lanes ? 16 / C.lanes : 32;  // rows of a group (by lanes two GPU lanes an entry lane)
    for (int q = 0; q < nr;) {
        const int l = C.level[C.row(rows[q])];
        int e = q;
        while (e < nr && e - q < most && C.level[C.row(rows[e])] == l) ++e;
        gfirst.push_back(q);
        for (int k = q; k < e; ++k) grp[k] = (int)gfirst.size() - 1;
        q = e;
    }
    const int ng = (int)gfirst.size();
    gfirst.push_back(nr);
    // halo: the rows of other tiles read here, in (level, order)
    const std::vector<int> &hal = halo.row;
    const int nh = (int)hal.size(), nch = (nh + 31) / 32;
    for (int q = 0; q < nh; ++q) S.hpos[hal[q]] = q;
    // first group that needs a chunk delivered, were every halo entry read through the ring
    std::vector<int> first_need((size_t)nch + 1, ng), wmark((size_t)ng, 0);
    for (int g = 0, run = 0; g < ng; ++g) {
        for (int q = gfirst[g]; q < gfirst[g + 1]; ++q) {
            const int i = C.row(rows[q]), t = C.ipos[i];
            for (int k = C.prp[t]; k < C.prp[t + 1]; ++k) {
                const int j = C.pci[k];
                if (j != i && C.ord(j) < p0) run = std::max(run, S.hpos[j] / 32 + 1);
            }
        }
        for (int c = (g ? wmark[g - 1] : 0); c < run; ++c) first_need[c] = g;
        wmark[g] = run;
    }
    // the last ring read of each own value and each halo value
    std::vector<int> own_last((size_t)nr, -1), halo_last((size_t)nh, -1);
    std::deque<int> live;                    // groups whose records are in the ring, oldest first
    std::vector<int> roff((size_t)ng), rsize((size_t)ng);
    int ring = 0;
    std::vector<Entry> ent;
    std::vector<int> of_row;                 // entries of the group's rows: [ptr[r], ptr[r + 1])
    std::vector<unsigned char> stage_of;     // 0 columns, 1 and 2 tails
    std::vector<int> far_of;                 // row of a far entry, -1
    std::vector<int> need_of;
    std::vector<int> code_of;
    int kt[3];
    for (int g = 0; g < ng; ++g) {
        const int q0 = gfirst[g], c = gfirst[g + 1] - q0;
        ent.clear();
        of_row.assign(1, 0);
        for (int r = 0; r < c; ++r) {
            const int i = C.row(rows[q0 + r]), t = C.ipos[i];
            for (int k = C.prp[t]; k < C.prp[t + 1]; ++k)
                if (C.pci[k] != i) ent.push_back({C.level[C.pci[k]], C.pci[k], k});
            // by age; by lanes the entries stay in column order
            if (!C.lanes)
                std::sort(ent.begin() + of_row[r], ent.end(), [&](const Entry &a, const Entry &b) {
                    return a.lev != b.lev ? a.lev < b.lev : C.ord(a.j) < C.ord(b.j);
                });
            of_row.push_back((int)ent.size());
        }
        stage_of.assign(ent.size(), 0);
        code_of.assign(ent.size(), 0);
        need_of.assign(ent.size(), 0);
        far_of.assign(ent.size(), -1);
        int own_need[3] = {-1, -1, -1}, halo_need[3] = {0, 0, 0};
        int K0 = 0;
        bool any_far = false;
        kt[1] = kt[2] = 0;
        const int lev = C.level[C.row(rows[q0])];
        for (int r = 0; r < c; ++r) {
            int k0 = 0, kr[3] = {0, 0, 0};
            for (int e = of_row[r]; e < of_row[r + 1]; ++e) {
                const int j = ent[e].j, d = lev - ent[e].lev;
                const bool own = C.ord(j) >= p0;
                bool far;
                int need = 0;
                if (own) {
                    const int q = pos[C.ord(j) - p0];
                    far = q + L.S_own < nr && g >= grp[q + L.S_own];
                    code_of[e] = q % L.S_own;
                    need = grp[q];
                    if (!far) own_last[q] = g;
                } else {
                    const int q = S.hpos[j];
                    const long long over = (long long)q + L.S_halo;
                    far = over < nh && g >= first_need[over / 32];
                    code_of[e] = L.S_own + q % L.S_halo;
                    need = q + 1;
                    if (!far) halo_last[q] = g;
                }
                int s = !C.lanes && d <= TS_TAILS ? TS_TAILS + 1 - d : 0;
                if (s && kr[s] >= TS_TAIL) s = 0;
                if (far) {
                    if (s) {
                        O.why = "a newest dependency left its ring";
                        break;
                    }
                    code_of[e] = TS_FAR;
                    far_of[e] = j;
                    any_far = true;
                    ++O.nfar;
                    ++k0;
                    continue;
                }
                stage_of[e] = (unsigned char)s;
                need_of[e] = need;
                if (s == 0) {
                    ++k0;
                    continue;
                }
                ++kr[s];
                if (own) own_need[s] = std::max(own_need[s], need);
                else halo_need[s] = std::max(halo_need[s], need);
            }
            K0 = std::max(K0, k0);
            for (int s = 1; s <= TS_TAILS; ++s) kt[s] = std::max(kt[s], kr[s]);
        }
        if (O.why) break;
        // the group overwrites the own-ring slots of its rows: their last readers first
        for (int q = q0; q < q0 + c; ++q)
            if (q >= L.S_own) own_need[TS_TAILS] = std::max(own_need[TS_TAILS], own_last[q - L.S_own]);
        // lanes a row in the columns: two where they fit (half the columns for one more addition)
        int lg = 0;
        if (C.lanes) lg = C.lanes == 4 ? 2 : 3;
        else if (c <= 16 && K0 > 2) lg = 1;
        const int G = 1 << lg, blk = C.lanes ? 1 : 4;
        const int D0 = (K0 + G - 1) / G, KT = kt[1] + kt[2], nb = (D0 + blk - 1) / blk;
        if (nb > 65535) {
            O.why = "a row with too many entries";
            break;
        }
        int KP = 0;
        for (int r = 0; r < c; ++r) KP = std::max(KP, pushes.count(rows[q0 + r]));
        const TileRec R = tile_rec(c, nb, blk, any_far, KT, KP, elem);
        if (R.size > L.B_rec / 2) {
            O.why = "a group's record does not fit the staging ring";
            break;
        }
        // place in the ring: the groups whose bytes it takes must be done
        int need = g - TS_NM;
        auto drop = [&]() {
            need = std::max(need, live.front());
            live.pop_front();
        };
        if (ring + R.size > L.B_rec) {
            // what the previous lap left behind this lap's end is older than what it left at the start
            while (!live.empty() && roff[live.front()] >= ring) drop();
            ring = 0;
        }
        while (!live.empty() && roff[live.front()] < ring + R.size && roff[live.front()] + rsize[live.front()] > ring)
            drop();
        roff[g] = ring;
        rsize[g] = R.size;
        live.push_back(g);
        const size_t base = O.rec.size();
        O.groups.push_back((int)(base / 16));
        O.groups.push_back(R.size / 16);
        O.groups.push_back(ring / 16);
        O.groups.push_back(std::max(need, -1));
        ring += R.size;
        O.rec.resize(base + (size_t)R.size, 0);
        unsigned char *rec = O.rec.data() + base;
        int *hd = (int *)rec;
        hd[0] = c | lg << 8 | kt[1] << 16 | kt[2] << 20;
        hd[1] = nb | (any_far ? 1 << 16 : 0);
        hd[2] = q0 % L.S_own;
        hd[3] = D0 - blk * (nb - 1);
        for (int s = 1; s <= TS_TAILS; ++s) {
            hd[2 + 2 * s] = own_need[s];
            hd[3 + 2 * s] = halo_need[s];
        }
        hd[8] = KP;
        hd[9] = R.o_push / 16;
        hd[12] = R.o_old / 16 | R.o_tail / 16 << 16;
        hd[13] = R.o_cold / 16 | R.o_ctail / 16 << 16;
        hd[14] = R.o_cfar / 16;
        hd[15] = R.o_row / 16 | R.o_lv / 16 << 16;
        int *need_b = (int *)(rec + R.o_need);
        for (int q = 0; q < nb; ++q) need_b[2 * q] = -1;
        int *rid = (int *)(rec + R.o_row), *cfar = (int *)(rec + R.o_cfar);
        unsigned short *cold = (unsigned short *)(rec + R.o_cold), *ctail = (unsigned short *)(rec + R.o_ctail);
        const unsigned short pad = (unsigned short)(L.S_own + L.S_halo);
        for (int q = 0; q < 32 * blk * nb; ++q) cold[q] = pad;
        for (int q = 0; q < 32 * KT; ++q) ctail[q] = pad;
        int *push = (int *)(rec + R.o_push);
        for (int q = 0; q < 32 * KP; ++q) push[q] = -1;
        for (int r = 0; r < c; ++r)
            for (int k = 0, m = pushes.count(rows[q0 + r]); k < m; ++k)
                push[32 * k + r] = pushes.dat[pushes.ptr[rows[q0 + r] - pushes.p0] + k];
        const int e_old = (int)((base + R.o_old) / elem), e_tail = (int)((base + R.o_tail) / elem),
                  e_lv = (int)((base + R.o_lv) / elem);
        for (int r = 0; r < c; ++r) {
            const int i = C.row(rows[q0 + r]), t = C.ipos[i];
            rid[r] = i;
            C.dlv[t] = e_lv + r;
            for (int k = C.prp[t]; k < C.prp[t + 1]; ++k)
                if (C.pci[k] == i) C.dval[k] = -1;
            // by age right-aligned: a short row's entries are as recent as the others' last ones
            int k0 = C.lanes ? 0 : 4 * nb * G, kr[3] = {0, 0, kt[1]};
            for (int e = of_row[r]; e < of_row[r + 1] && !C.lanes; ++e) k0 -= stage_of[e] == 0;
            for (int e = of_row[r]; e < of_row[r + 1]; ++e) {
                if (stage_of[e] == 0) {
                    const int q = k0 / G, lane = r * G + k0 % G, b = q / blk;
                    if (far_of[e] < 0) {
                        int &m = need_b[2 * b + (C.ord(ent[e].j) < p0)];
                        m = std::max(m, need_of[e]);
                    } else {
                        cfar[32 * blk * b + blk * lane + q % blk] = far_of[e];
                    }
                    cold[32 * blk * b + blk * lane + q % blk] = (unsigned short)code_of[e];
                    C.dval[ent[e].k] = e_old + 32 * blk * b + ts_col(q % blk, lane, blk, elem);
                    ++k0;
                } else {
                    const int at = kr[stage_of[e]]++ * 32 + r;
                    ctail[at] = (unsigned short)code_of[e];
                    C.dval[ent[e].k] = e_tail + at;
                }
            }
        }
    }
    // halo values: rows, and the group after whose end the slots' previous values are dead
    O.halo.assign((size_t)nch * 32, -1);
    O.rel.assign((size_t)nch, -1);
    for (int q = 0; q < nh; ++q) {
        O.halo[q] = halo.pushed[q] ? -2 : hal[q];
        if (q >= L.S_halo) O.rel[q / 32] = std::max(O.rel[q / 32], halo_last[q - L.S_halo]);
    }
    for (int h : hal) S.hpos[h] = -1;
}

int plan_threads() {
    if (const char *e = std::getenv("SSG_PLAN_THREADS")) {
        const int v = std::atoi(e);
        if (v >= 1 && v <= 64) return v;
    }
    const unsigned hc = std::thread::hardware_concurrency();
    return (int)std::max(1u, std::min(16u, hc / 2));
}

}  // namespace

TilePlanHost tile_plan_host(int n, int nlev, const int *prp, const int *pci, const int *ipos, const int *level,
                            bool lower, int elem, int lanes, int T, int CS, const TileLayout *lay,
                            const TileLimits *lim) {
    TilePlanHost P;
    auto fail = [&](const char *why) {
        P.ok = false;
        P.why = why;
        return P;
    };
    if (n <= 0) return fail("no rows");
    if (lanes != 0 && lanes != 4 && lanes != 8) return fail("not a number of lanes a row the records hold");
    if (T <= 0) T = tile_count(n, lanes);
    T = std::min(T, n);
    P.T = T;
    P.CS = CS = std::max(1, CS);
    P.lay = lay ? *lay : tile_layout(elem, lanes);
    P.dval.assign((size_t)prp[n], -1);
    P.dlv.assign((size_t)n, 0);
    auto first = [&](int t) { return (int)((long long)n * t / T); };
    // four passes: over tiles, clusters, tiles, and tiles again to put the outputs in their places, which are known once every
    // tile is planned; items are taken one at a time by a few host threads. (With the last pass on one thread 80^3 took 144 ms
    // forward and 233 backward, now 95 and 136.)
    const int nt = std::max(1, std::min(plan_threads(), T)), NC = (T + CS - 1) / CS;
    const int items[4] = {T, CS > 1 ? NC : 0, T, T};
    std::vector<Halo> halo((size_t)T);
    std::vector<Push> push((size_t)NC);
    std::vector<TileOut> out((size_t)T);
    const Ctx C{n, elem, lanes, prp, pci, ipos, level, lower, P.lay, P.dval.data(), P.dlv.data()};
    std::atomic<int> next[4] = {{0}, {0}, {0}, {0}}, done[4] = {{0}, {0}, {0}, {0}};
    std::vector<std::exception_ptr> errs((size_t)nt);
    // a limit passed: the passes run out without work. Each limit is on a maximum or a sum, so the outcome does not depend on
    // the threads.
    std::atomic<const char *> over{nullptr};
    std::atomic<long long> nfar{0}, bytes{0};
    const double max_chunks = lim ? lim->chunks_per_level * std::max(nlev, 1) : 0.0;
    const double max_far = lim ? lim->far_per_row * n : 0.0;
    // places of the tiles' outputs, or why there is no plan
    const char *why = nullptr;
    auto place = [&]() {
        for (int t = 0; t < T && !why; ++t) why = halo[t].why;
        if (!why) why = over.load();
        for (int t = 0; t < T && !why; ++t) why = out[t].why;
        for (auto &e : errs)
            if (e) why = "an exception";  // thrown below
        if (why) return;
        for (auto &p : push) P.npush += (int)p.dat.size();
        long long off = 0, g0 = 0, c0 = 0;
        P.tiles.resize((size_t)T * 4);
        P.rec.resize((size_t)T);
        P.rec_off.resize((size_t)T + 1);
        for (int t = 0; t < T; ++t) {
            P.rec_off[t] = off;
            P.tiles[4 * t] = (int)g0;
            P.tiles[4 * t + 1] = (int)out[t].groups.size() / 4;
            P.tiles[4 * t + 2] = (int)c0;
            P.tiles[4 * t + 3] = (int)out[t].rel.size();
            g0 += (long long)out[t].groups.size() / 4;
            c0 += (long long)out[t].rel.size();
            off += (long long)out[t].rec.size();
            P.nfar += out[t].nfar;
        }
        P.rec_off[T] = off;
        P.rec_bytes = off;
        if (off / elem >= (1ll << 31) || g0 >= (1ll << 29) || c0 >= (1ll << 26)) {
            why = "records too large";
            return;
        }
        P.groups.resize((size_t)g0 * 4);
        P.halo.resize((size_t)c0 * 32);
        P.rel.resize((size_t)c0);
    };
    auto put = [&](int t) {
        const int r16 = (int)(P.rec_off[t] / 16), rel_e = (int)(P.rec_off[t] / elem);
        TileOut &o = out[t];
        for (size_t q = 0; q < o.groups.size(); q += 4) o.groups[q] += r16;
        std::copy(o.groups.begin(), o.groups.end(), P.groups.begin() + (size_t)P.tiles[4 * t] * 4);
        std::copy(o.halo.begin(), o.halo.end(), P.halo.begin() + (size_t)P.tiles[4 * t + 2] * 32);
        std::copy(o.rel.begin(), o.rel.end(), P.rel.begin() + (size_t)P.tiles[4 * t + 2]);
        for (int p = first(t); p < first(t + 1); ++p) {
            const int i = lower ? p : n - 1 - p, q = ipos[i];
            P.dlv[q] += rel_e;
            for (int k = prp[q]; k < prp[q + 1]; ++k)
                if (P.dval[k] >= 0) P.dval[k] += rel_e;
        }
        P.rec[t] = std::move(o.rec);
    };
    std::atomic<int> placed{0};
    auto work = [&](int q) {
        std::unique_ptr<Scratch> S;
        for (int pass = 0; pass < 4; ++pass) {
            if (pass == 3) {
                if (q == 0) {
                    try {
                        place();
                    } catch (...) {
                        errs[q] = std::current_exception();
                        why = "an exception";
                    }
                    placed = 1;
                }
                while (!placed.load()) std::this_thread::yield();
                if (why) return;
            }
            for (int t; (t = next[pass].fetch_add(1)) < items[pass]; done[pass].fetch_add(1)) {
                try {
                    if (over.load()) continue;
                    if (!S) S.reset(new Scratch(n));
                    if (pass == 0) {
                        find_halo(C, first(t), first(t + 1), *S, halo[t]);
                        if (lim && (double)((halo[t].row.size() + 31) / 32) > max_chunks)
                            over = "a tile reads too many rows of others";
                    } else if (pass == 1) {
                        find_pushes(C, t * CS, std::min(T, (t + 1) * CS), first, halo, push[t]);
                    } else if (pass == 3) {
                        put(t);
                    } else if (!halo[t].why) {
                        plan_tile(C, first(t), first(t + 1), halo[t], push[t / CS], *S, out[t]);
                        if (lim && (double)(nfar += out[t].nfar) > max_far) over = "too many far entries";
                        if (lim && (bytes += (long long)out[t].rec.size()) > lim->bytes) over = "records too large";
                    }
                } catch (...) {
                    errs[q] = std::current_exception();
                }
            }
            while (done[pass].load() < items[pass]) std::this_thread::yield();
        }
    };
    std::vector<std::thread> pool;
    for (int q = 1; q < nt; ++q) {
        try {
            pool.emplace_back(work, q);
        } catch (...) {
            break;  // fewer threads: the others take its items
        }
    }
    work(0);
    for (auto &t : pool) t.join();
    for (auto &e : errs)
        if (e) std::rethrow_exception(e);
    if (why) return fail(why);
    P.ok = true;
    return P;
}

}  // namespace ssg
