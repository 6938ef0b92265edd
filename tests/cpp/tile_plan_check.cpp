// Checks and emulates the tile sweep's host plan (ss_tile_plan.cpp) for tests/test_tile_plan.py, independently of the
// plan's own reasoning: every read's source, every ring reuse and every wait, then the sums themselves.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "ss_tile_plan.hpp"

using namespace ssg;

static std::string bad(const char *what, int tile, int g, int x) {
    char s[200];
    std::snprintf(s, sizeof s, "%s (tile %d, group %d, %d)", what, tile, g, x);
    return s;
}

// values of the triangle in its level-ordered layout, lvec per level-ordered row, rhs by row; y: the solution.
// lay: {S_own, S_halo, B_rec} or null. Returns "" or what is wrong; stats: tiles, far entries.
static std::string run(int n, int nlev, const int *prp, const int *pci, const int *ipos, const int *level, bool lower,
                       int lanes, int T, int CS, const int *lay, const double *val, const double *lvec, const double *rhs, double *y,
                       int *stats) {
    TileLayout L = tile_layout(8, lanes);
    if (lay) {
        L.S_own = lay[0];
        L.S_halo = lay[1];
        L.B_rec = lay[2];
    }
    const TilePlanHost P = tile_plan_host(n, nlev, prp, pci, ipos, level, lower, 8, lanes, T, CS, &L);
    if (!P.ok) return std::string("no plan: ") + P.why;
    if (L.o_rec + (lay ? 0 : L.B_rec) > TS_SMEM_MAX) return "layout exceeds shared memory";
    stats[0] = P.T;
    stats[1] = P.nfar;
    // the records with their values, as k_tile_fill leaves them
    std::vector<unsigned char> rec((size_t)P.rec_bytes + 16, 0);
    for (int t = 0; t < P.T; ++t)
        if (!P.rec[t].empty()) std::memcpy(rec.data() + P.rec_off[t], P.rec[t].data(), P.rec[t].size());
    double *rv = (double *)rec.data();
    std::vector<char> hit((size_t)prp[n], 0);
    for (int q = 0; q < n; ++q) {
        rv[P.dlv[q]] = lvec[q];
        for (int k = prp[q]; k < prp[q + 1]; ++k)
            if (P.dval[k] >= 0) rv[P.dval[k]] = lanes ? -val[k] : -(val[k] * lvec[q]);
    }
    std::vector<char> done((size_t)n, 0);
    int rows_seen = 0;
    std::vector<std::vector<int>> slots((size_t)CS);  // rows pushed to each CTA of the cluster, by slot
    for (int t = 0; t < P.T; ++t) {
        const int g0 = P.tiles[4 * t], ng = P.tiles[4 * t + 1], c0 = P.tiles[4 * t + 2], nch = P.tiles[4 * t + 3];
        std::vector<int> own_row, own_grp;           // by production position
        std::vector<std::vector<int>> own_rd, halo_rd((size_t)nch * 32);  // groups that read each value from its ring
        std::vector<int> need3((size_t)ng), hneed((size_t)ng, 0);
        if (t % CS == 0)
            for (auto &v : slots) v.assign((size_t)L.S_halo, -1);
        std::vector<int> hrow((size_t)nch * 32);
        for (int c = 0; c < nch * 32; ++c) {
            int j = P.halo[(size_t)c0 * 32 + c];
            if (j == -2) {
                j = c < L.S_halo ? slots[t % CS][c] : -1;
                if (j < 0) return bad("a halo value is not pushed", t, c, j);
            } else if (c < L.S_halo && slots[t % CS][c] >= 0) {
                return bad("a push nobody reads", t, c, j);
            }
            hrow[c] = j;
            if (j >= 0 && !done[j]) return bad("a halo value of a later tile", t, c, j);
            if (c && j >= 0 && level[j] < level[hrow[c - 1]]) return bad("halo order", t, c, j);
        }
        struct Span { int o, e; };
        std::vector<Span> span;
        int staged = -1;
        std::vector<int> tile_rows;
        for (int g = 0; g < ng; ++g) {
            const int *gm = &P.groups[(size_t)(g0 + g) * 4];
            const unsigned char *r = rec.data() + 16ll * gm[0];
            const int *hd = (const int *)r;
            const int cnt = hd[0] & 0xff, lg = (hd[0] >> 8) & 0xff, G = 1 << lg;
            const int kt[3] = {0, (hd[0] >> 16) & 15, (hd[0] >> 20) & 15};
            const int nb = hd[1] & 0xffff, blk = lanes ? 1 : 4;
            const bool far = (hd[1] >> 16) != 0;
            const TileRec R = tile_rec(cnt, nb, blk, far, kt[1] + kt[2], hd[8], 8);
            if (cnt < 1 || cnt * G > (lanes ? 16 : 32)) return bad("group shape", t, g, cnt);
            if (R.size != 16 * gm[1] || 16 * gm[2] + R.size > L.B_rec) return bad("record size", t, g, R.size);
            // the staging ring: whoever's bytes it takes must be done, and the barrier slot free
            const Span me{16 * gm[2], 16 * gm[2] + R.size};
            staged = std::max(staged, gm[3]);  // copies are issued in order, so earlier copies' waits hold too
            for (int o = 0; o < g; ++o)
                if (o > staged && span[o].o < me.e && span[o].e > me.o) return bad("record ring overlap", t, g, o);
            if (gm[3] >= g || staged < g - TS_NM) return bad("staging wait", t, g, gm[3]);
            span.push_back(me);
            const int q0 = (int)own_row.size();
            if (hd[2] != q0 % L.S_own) return bad("own slot", t, g, hd[2]);
            const int *rid = (const int *)(r + R.o_row);
            const unsigned short *cold = (const unsigned short *)(r + R.o_cold), *ct = (const unsigned short *)(r + R.o_ctail);
            const int *cf = (const int *)(r + R.o_cfar);
            const double *vo = (const double *)(r + R.o_old), *vt = (const double *)(r + R.o_tail), *lv = (const double *)(r + R.o_lv);
            // waits: the tail stages, then the blocks of columns
            std::vector<int> own_w{hd[4], hd[6]}, halo_w{hd[5], hd[7]};
            if (nb && (hd[3] < 1 || hd[3] > blk)) return bad("first block", t, g, hd[3]);
            for (int q = 0; q < nb; ++q) {
                own_w.push_back(((const int *)(r + R.o_need))[2 * q]);
                halo_w.push_back(((const int *)(r + R.o_need))[2 * q + 1]);
            }
            for (size_t w = 0; w < own_w.size(); ++w) {
                if (own_w[w] >= g) return bad("a group waits for itself or a later one", t, g, own_w[w]);
                if (halo_w[w] > 32 * nch) return bad("halo wait", t, g, halo_w[w]);
                hneed[g] = std::max(hneed[g], halo_w[w]);
            }
            need3[g] = own_w[TS_TAILS - 1];
            if (hd[12] != (R.o_old / 16 | R.o_tail / 16 << 16) || hd[13] != (R.o_cold / 16 | R.o_ctail / 16 << 16) ||
                hd[14] != R.o_cfar / 16 || hd[9] != R.o_push / 16 || hd[15] != (R.o_row / 16 | R.o_lv / 16 << 16))
                return bad("record offsets", t, g, 0);
            std::vector<double> res((size_t)cnt);
            for (int i = 0; i < cnt; ++i) {
                const int row = rid[i];
                if (row < 0 || row >= n || done[row]) return bad("row", t, g, row);
                // what ring slot `code` holds for this reader, checked against the stage's waits
                std::string why;
                auto read = [&](int code, int s) -> double {
                    if (code == L.S_own + L.S_halo) return 0.0;
                    if (code < L.S_own) {
                        int q = -1;  // the newest value in the slot
                        for (int p = code; p < q0; p += L.S_own) q = p;
                        if (q < 0 || own_grp[q] > own_w[s]) why = bad("own value not waited for", t, g, q);
                        else own_rd[q].push_back(g);
                        return q < 0 ? 0.0 : y[own_row[q]];
                    }
                    // halo: the newest chunk the waits let through; none newer may have come (checked below)
                    int q = -1;
                    for (int p = code - L.S_own; p < halo_w[s] && p < 32 * nch; p += L.S_halo)
                        if (hrow[p] >= 0) q = p;  // padding lanes write nothing
                    if (q < 0) why = bad("halo value not waited for", t, g, code);
                    else halo_rd[q].push_back(g);
                    return q < 0 ? 0.0 : y[hrow[q]];
                };
                double s0 = 0.0;
                for (int q = 0; q < blk * nb; ++q)
                    for (int l = i * G; l < i * G + G; ++l) {
                        const int at = 32 * blk * (q / blk), code = cold[at + blk * l + q % blk];
                        if (!lanes && q < 4 - hd[3] && code != L.S_own + L.S_halo) return bad("a skipped column", t, g, q);
                        const double a = vo[at + ts_col(q % blk, l, blk, 8)];
                        if (code == TS_FAR) {
                            const int j = far ? cf[at + blk * l + q % blk] : -1;
                            if (j < 0 || j >= n || !done[j]) return bad("far value not done", t, g, j);
                            s0 += a * y[j];
                        } else {
                            s0 += a * read(code, TS_TAILS + q / blk);
                        }
                    }
                double v = lanes ? (rhs[row] + s0) * lv[i] : rhs[row] * lv[i] + s0;
                for (int s = 1, k = 0; s <= TS_TAILS; ++s)
                    for (int q = 0; q < kt[s]; ++q, ++k) v += vt[k * 32 + i] * read(ct[k * 32 + i], s - 1);
                if (!why.empty()) return why;
                res[i] = v;
            }
            for (int k = 0; k < 32 * hd[8]; ++k) {
                const int w = ((const int *)(r + R.o_push))[k];
                if (w < 0) continue;
                const int to = w >> 20, slot = w & 0xfffff;
                if (k % 32 >= cnt || to <= t % CS || to >= CS || t - t % CS + to >= P.T || slot >= L.S_halo || slots[to][slot] >= 0)
                    return bad("push", t, g, w);
                slots[to][slot] = rid[k % 32];
            }
            for (int i = 0; i < cnt; ++i) {
                y[rid[i]] = res[i];
                own_row.push_back(rid[i]);
                own_grp.push_back(g);
                own_rd.emplace_back();
                tile_rows.push_back(rid[i]);
            }
            for (int i = 0; i < cnt; ++i) done[rid[i]] = 1;
            rows_seen += cnt;
        }
        // own ring: a slot's readers are done before its next writer writes
        for (int q = 0; q + L.S_own < (int)own_row.size(); ++q)
            for (int u : own_rd[q])
                if (u > need3[own_grp[q + L.S_own]]) return bad("own slot rewritten too early", t, own_grp[q + L.S_own], u);
        // halo ring: likewise for a chunk's delivery, and no chunk waits for a group that needs it
        for (int q = 0; q + L.S_halo < nch * 32 && hrow[q + L.S_halo] >= 0; ++q)
            for (int u : halo_rd[q])
                if (u > P.rel[(size_t)c0 + (q + L.S_halo) / 32]) return bad("halo slot rewritten too early", t, u, q);
        for (int g = 0, run = 0; g < ng; ++g) {
            for (int c = run; c < hneed[g]; ++c)
                if (P.rel[(size_t)c0 + c / 32] >= g) return bad("a chunk waits for a group that needs it", t, g, c);
            run = std::max(run, hneed[g]);
        }
    }
    return rows_seen == n ? "" : "rows missing";
}

extern "C" const char *tile_check(int n, int nlev, const int *prp, const int *pci, const int *ipos, const int *level,
                                  int lower, int lanes, int T, int CS, const int *lay, const double *val, const double *lvec,
                                  const double *rhs, double *y, int *stats) {
    static std::string why;
    why = run(n, nlev, prp, pci, ipos, level, lower != 0, lanes, T, CS, lay, val, lvec, rhs, y, stats);
    return why.c_str();
}
