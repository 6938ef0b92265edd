// ss_tile.cu -- whole-GPU tile sweeps for every triangular solve of the solvers:
// the IC pair of MatSolverBase::IC_frbc_process (src/MatSolverBase.cpp:177-231),
// fr_process / bc_process (:243-327) and the Eisenstat sweep of
// MatSolverMRTR_SGSver.cpp:187-189.
//
// A sweep is bound by its dependency levels, not by bytes. The schedule
// (ss_tile_plan.hpp) cuts the rows into tiles of consecutive rows; a CTA owns a
// tile, so all but the tile borders of a dependency path stay inside one SM, and
// because tiles only depend on lower tiles, the latency of a border is paid once
// per border and not once per level.
//
// By age, 8 consecutive tiles run on one thread-block cluster and store what they
// solve into the rings of the cluster's CTAs that read it (st.relaxed.cluster): a
// border inside the cluster costs a store into another SM and a poll of the own
// shared memory in place of a store to memory and polls of the L2. The first lap of
// a ring is filled that way, whose slots the CTA marks unsolved before the cluster's
// barrier lets anyone start; later laps and other clusters' values come from memory.
//
// A cluster claims its tiles in order through a ticket (every wait is on a tile some
// running cluster holds, or of the same cluster) and its CTAs run three kinds of warps:
//   * compute warps take the tile's groups round robin (group g: warp g % TS_W),
//     sum, write the values to the own ring, publish their progress and store the
//     values to the cluster's readers and to memory;
//   * receiver warps bring the halo in, 32 values a chunk: each lane polls the
//     output vector for one value (a sentinel marks the unsolved) and puts it into
//     the halo ring, or polls the ring for a value the cluster stores there; the
//     count of values here, in list order, is published;
//   * one warp stages the groups' records with bulk copies as ring space frees.
// Waits inside a CTA are one load of the progress words, one vote and a warp barrier.
// Values go between CTAs one aligned 4- or 8-byte store at a time, which is
// single-copy atomic, so a value is its own flag and no fence is needed.
//
// What bounds it: the chain of dependency levels (1,410 forward at 80^3), not bytes
// (1 % of HBM) and not yet FP64: an FP64 instruction holds its warp for 64 cycles
// and an SM issues one in 19, so a group's 12-15 instructions set the split of the
// sums. Measured on a GB300, microseconds a sweep (forward / backward), with the
// one-cluster schedules this replaces as the automatic choice in brackets:
//   curl-curl, real:  10^3  54 / 55 [221 / 222], 20^3 120 / 123 [496 / 501],
//                     41^3 322 / 325 [1,095 / 1,090], 80^3 908 / 904 [2,237 / 2,195] (push); without clusters 123 / 127,
//                     375 / 379 and 1,101 / 994
//   SGS pair, 48^3:   439 / 417 [1,834 / 1,810] (lockstep)
//   eddy currents:    33^3 640 / 813 [1,638 / 1,525], 60^3 1,310 / 1,668 [3,616 / 3,338] (lockstep); 707 / 903 and
//                     1,490 / 1,830 with a lane holding both parts of a sum and 2.5 times fewer tiles
//   FP32, 44^3:       206 / 210 [504 / 498] (push)
//
// Every wait is bounded (the handle's spin limit) and ends early when the error
// word is set; the CTA then drains its copies and only goes along to the cluster's
// barriers, until its cluster leaves together.
#include <algorithm>
#include <exception>
#include <new>
#include <thread>
#include <utility>
#include <vector>

#include "sparsesolv_gb300.h"
#include "ss_internal.cuh"
#include "ss_krylov.cuh"

namespace ssg {

// ---------------------------------------------------------------- device helpers
__device__ __forceinline__ void tl_mbar_init(unsigned a, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void tl_mbar_inval(unsigned a) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void tl_mbar_expect(unsigned a, unsigned tx) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(tx) : "memory");
}
__device__ __forceinline__ bool tl_mbar_test(unsigned a, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tl_bulk_g2s(unsigned dst, const void *src, unsigned bytes, unsigned mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void tl_st_release(unsigned a, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ int tl_ld_acquire(unsigned a) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// one value of the output vector, written by any CTA: false while unsolved
__device__ __forceinline__ bool tl_take(const double *p, double &v) {
    v = ld_vol(p);
    return !is_sent(v);
}
__device__ __forceinline__ bool tl_take(const float *p, float &v) {
    v = ld_vol(p);
    return !is_sent(v);
}
__device__ __forceinline__ bool tl_take(const cplx *p, cplx &v) {
    v.x = ld_vol(&p->x);
    v.y = ld_vol(&p->y);
    return !is_sent(v.x) && !is_sent(v.y);
}
__device__ __forceinline__ bool tl_take(const cplxf *p, cplxf &v) {
    v.x = ld_vol(&p->x);
    v.y = ld_vol(&p->y);
    return !is_sent(v.x) && !is_sent(v.y);
}
__device__ __forceinline__ void tl_give(double *p, double v) { st_vol(p, unsent(v)); }
__device__ __forceinline__ void tl_give(float *p, float v) { st_vol(p, unsent(v)); }
__device__ __forceinline__ void tl_give(cplx *p, cplx v) {
    st_vol(&p->x, unsent(v.x));
    st_vol(&p->y, unsent(v.y));
}
__device__ __forceinline__ void tl_give(cplxf *p, cplxf v) {
    st_vol(&p->x, unsent(v.x));
    st_vol(&p->y, unsent(v.y));
}

// CTAs of a cluster: a value stored into another one's shared memory, and barriers of all
__device__ __forceinline__ unsigned tl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned tl_mapa(unsigned a, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void tl_send(unsigned a, int v) {
    asm volatile("st.relaxed.cluster.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void tl_send(unsigned a, float v) {
    asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(unsent(v)) : "memory");
}
__device__ __forceinline__ void tl_send(unsigned a, double v) {
    asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(unsent(v)) : "memory");
}
__device__ __forceinline__ void tl_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

static_assert(TS_NM % TS_W == 0, "groups of one barrier belong to one warp");
static_assert(TS_TAILS == 2 && TS_W < 32, "the stages and progress words below");

// one lane's four values of a block of columns (ts_col)
__device__ __forceinline__ void tl_vals(const double *b, int lane, double (&v)[4]) {
    const double2 p = ((const double2 *)b)[lane], q = ((const double2 *)b)[32 + lane];
    v[0] = p.x, v[1] = p.y, v[2] = q.x, v[3] = q.y;
}
__device__ __forceinline__ void tl_vals(const float *b, int lane, float (&v)[4]) {
    const float4 p = ((const float4 *)b)[lane];
    v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = p.w;
}
__device__ __forceinline__ void tl_vals(const cplx *b, int lane, cplx (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 p = ((const double2 *)b)[32 * q + lane];
        v[q] = {p.x, p.y};
    }
}
__device__ __forceinline__ void tl_vals(const cplxf *b, int lane, cplxf (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
        const float4 p = ((const float4 *)b)[16 * q + lane];
        v[q] = {p.x, p.y};
        v[q + 1] = {p.z, p.w};
    }
}

struct TileArgs {
    int T, CS;
    const int4 *tiles, *groups;
    const int *halo, *rel;
    const unsigned char *rec;
    const void *rhs, *aux;
    void *out, *out2;
    int *ticket;   // zero at launch
    const KState *st;
    int *err;
    TileLayout L;
};

// the time limit of a wait, looked at every so many polls
struct Bound {
    int *err;
    unsigned long long lim, t0 = 0;
    unsigned polls = 0;
    __device__ Bound(int *e, unsigned long long l) : err(e), lim(l) {}
    // true: give up
    __device__ __forceinline__ bool spent(unsigned mask) {
        if ((++polls & mask) != 0) return false;
        if (*(volatile int *)err) return true;
        const unsigned long long t = gtimer();
        if (t0 == 0) t0 = t;
        if (t - t0 > lim) {
            atomicExch(err, ERR_TIMEOUT);
            return true;
        }
        return false;
    }
};

// LANES: 0 sums by age, 4 or 8 by lanes (ss_tile_plan.hpp)
// CL: clusters of several CTAs
template <typename T, int MODE, int LANES, bool CL>
__global__ void __launch_bounds__(TS_THREADS, 1) k_sweep_tile(TileArgs a) {
    if (a.st && !a.st->active) return;
    extern __shared__ __align__(16) unsigned char tl_smem[];
    __shared__ int s_tile;
    const TileLayout &L = a.L;
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(tl_smem);
    T *X = (T *)(tl_smem + L.o_x);
    int *place = (int *)(tl_smem + L.o_place);  // record ring offsets / 16 of the staged groups
    const unsigned full = sbase + L.o_full, prog = sbase + L.o_prog;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const T *rhs = (const T *)a.rhs, *aux = (const T *)a.aux;
    T *out = (T *)a.out, *out2 = (T *)a.out2;
    const unsigned long long lim = spin_limit_ns(a.err);
    constexpr int EB = (int)sizeof(T);
    bool bad = false;
    const int CS = CL ? a.CS : 1, rank = CL ? (int)tl_rank() : 0;
    const unsigned ring = sbase + (unsigned)L.o_x + (unsigned)(L.S_own * EB);  // the halo ring, here and in the other CTAs

    if (tid == 0) X[L.S_own + L.S_halo] = Sc<T>::zero();
    const bool once = a.T <= (int)gridDim.x;  // as many CTAs as tiles: each takes one
    for (bool first = true;; first = false) {
        // ---- next CS tiles, one a CTA
        int t = 0;
        if (tid == 0 && rank == 0 && (first || !CL)) t = atomicAdd(a.ticket, 1) * CS;
        if (!CL) {
            if (tid == 0) s_tile = t;
        } else {
            tl_cluster_sync();  // no CTA of the cluster stores into this one's ring any more
            if (rank == 0 && tid == 0) {
                // not before all of the cluster are done: another cluster may be free earlier (80^3: 966 us instead of 911)
                if (!first) t = *(volatile int *)a.err ? a.T : atomicAdd(a.ticket, 1) * CS;
                for (int q = 0; q < CS; ++q) tl_send(tl_mapa((unsigned)__cvta_generic_to_shared(&s_tile), q), t);
            }
            // slots of the first lap unsolved
            for (int q = tid; q < L.S_halo * EB / 16; q += TS_THREADS)
                ((uint4 *)(X + L.S_own))[q] = make_uint4(~0u, ~0u, ~0u, ~0u);
        }
        if (tid < TS_NM) tl_mbar_init(full + 8u * tid, 1);
        if (tid < 32) ((volatile int *)(tl_smem + L.o_prog))[tid] = tid < TS_W ? tid : 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!CL) __syncthreads();
        else tl_cluster_sync();
        if (s_tile >= a.T) break;
        const int tile = s_tile + rank;
        // a CTA without a tile goes along to the barriers, and so does one that gave up
        const int4 td = tile < a.T && !bad ? a.tiles[tile] : make_int4(0, 0, 0, 0);
        const int ng = td.y, nch = td.w;
        int issued = 0;  // groups staged

        // own groups up to og are done and h halo values are here. Lane w acquires what warp w released; the vote says that
        // all are here but orders no memory (CUDA promises that of __syncwarp alone), so the barrier is what lets every lane
        // read, or overwrite, what another lane acquired.
        auto ready = [&](int og, int h) {
            const int want = lane < TS_W ? og + 1 : lane == TS_W ? h : 0;
            const bool ok = __all_sync(0xffffffffu, tl_ld_acquire(prog + 4u * lane) >= want) != 0;
            if (ok) __syncwarp();
            return ok;
        };
        auto wait_for = [&](int og, int h) {
            if (ready(og, h)) return;
            Bound b(a.err, lim);
            while (!(ready(og, h) || ready(og, h) || ready(og, h)))
                if (__any_sync(0xffffffffu, b.spent(255))) {
                    bad = true;
                    return;
                }
        };
        // group g's record, once staged; null: give up. A warp that tests a staged group's barrier has itself taken the group
        // staged there before, so the parity is unambiguous.
        auto record = [&](int g) -> const unsigned char * {
            const unsigned bar = full + 8u * (g % TS_NM);
            const unsigned par = (unsigned)((g / TS_NM) & 1);
            // one loop of the whole warp, as everywhere here: lanes that leave loops of their own stay apart afterwards, and
            // each part of a warp takes the FP64 pipe for itself
            bad = __any_sync(0xffffffffu, bad);
            if (!bad && !__all_sync(0xffffffffu, tl_mbar_test(bar, par))) {
                Bound b(a.err, lim);
                while (!__all_sync(0xffffffffu, tl_mbar_test(bar, par)))
                    if (__any_sync(0xffffffffu, b.spent(255))) {
                        bad = true;
                        break;
                    }
            }
            return bad ? nullptr : tl_smem + L.o_rec + 16 * place[g % TS_NM];
        };

        if (warp < TS_W) {
            // ------------------------------------------------ compute warps
            for (int g = warp; g < ng; g += TS_W) {
                const unsigned char *rec = record(g);
                if (!rec) break;
                const int4 *hd = (const int4 *)rec;
                const int4 h0 = hd[0], nd = hd[1], hp = hd[2], of = hd[3];
                const int cnt = h0.x & 0xff, lg = (h0.x >> 8) & 0xff;
                const int nb = h0.y & 0xffff;
                const int *cfar = (h0.y >> 16) ? (const int *)(rec + 16 * of.z) : nullptr;
                const int2 *need = (const int2 *)(rec + 64);
                const T *v = (const T *)(rec + 16 * (of.x & 0xffff));
                // a column's value: from the rings, or from memory where its slot is reused too early
                auto value = [&](int code, const int *far_row) -> T {
                    T x = Sc<T>::zero();
                    bool have = code != TS_FAR;
                    if (have) x = X[code];
                    if (__all_sync(0xffffffffu, have)) return x;
                    const T *p = out + (have ? 0 : *far_row);
                    Bound b(a.err, lim);
                    do {
                        if (!have) have = tl_take(p, x);
                        if (__any_sync(0xffffffffu, b.spent(63))) {
                            bad = true;
                            break;
                        }
                    } while (!__all_sync(0xffffffffu, have));
                    return x;
                };
                int row = 0;
                bool lead;  // this lane has the row's result (or a component of it)
                // who else reads the row: the first two ahead, as the record is given back with the result
                const int *push = (const int *)(rec + 16 * hp.y);
                int to0 = -1, to1 = -1;
                auto send = [&](int to, auto val, int comp) {
                    if (CL && to >= 0)
                        tl_send(tl_mapa(ring + (unsigned)((to & 0xfffff) * EB + comp), (unsigned)to >> 20), val);
                };
                if constexpr (LANES > 0) {
                    // Lanes 2 l and 2 l + 1 hold the real and the imaginary part of entry lane l's sum. The arithmetic is
                    // that of k_sweep on complex values, a component a lane: the forward right-hand side starts lane 0's
                    // sum, the IC pair's values come negated.
                    using R = typename Sc<T>::real;
                    constexpr int W = 2 * LANES;  // GPU lanes a row
                    const int r = lane / W, el = lane >> 1;
                    const bool im = lane & 1;
                    lead = lane % W < 2 && r < cnt;
                    auto part = [&](T q) { return im ? q.y : q.x; };
                    // components of a * b and of acc + a * b: p, q the parts of b that a.x and a.y meet
                    auto cmul = [&](T f, R p, R q) { return mul_rn(f.x, p) + (im ? mul_rn(f.y, q) : -mul_rn(f.y, q)); };
                    auto cmadd = [&](R s, T f, R p, R q) {
                        if constexpr (sizeof(R) == 8) return fma(im ? f.y : -f.y, q, fma(f.x, p, s));
                        else return s + cmul(f, p, q);
                    };
                    R b0 = R(0), ua = R(0);
                    T lv = Sc<T>::zero();
                    if (lead) row = ((const int *)(rec + 16 * (of.w & 0xffff)))[r];
                    if (r < cnt) lv = ((const T *)(rec + 16 * ((unsigned)of.w >> 16)))[r];
                    if (lead) {
                        if (CL && hp.x > 0) to0 = push[r];
                        if (CL && hp.x > 1) to1 = push[32 + r];
                        if (MODE != SW_BWD_IC) b0 = part(rhs[row]);
                        if (MODE == SW_BWD_IC || MODE == SW_FWD_EIS) ua = part(aux[row]);
                    }
                    R acc = MODE == SW_FWD_DIV ? b0 : R(0);
                    const unsigned short *c = (const unsigned short *)(rec + 16 * (of.y & 0xffff)) + el;
                    v += el;
#pragma unroll 1
                    for (int k = 0; k < nb; ++k) {
                        const int2 w = need[k];
                        const int cc = c[32 * k];
                        const T vv = v[32 * k];
                        wait_for(w.x, w.y);
                        const T xx = cfar ? value(cc, cfar + 32 * k + el) : X[cc];
                        acc = cmadd(acc, vv, im ? xx.y : xx.x, im ? xx.x : xx.y);
                    }
#pragma unroll
                    for (int m = LANES / 2; m >= 1; m >>= 1) acc = acc + __shfl_xor_sync(0xffffffffu, acc, 2 * m);
                    R num = acc;
                    if (MODE == SW_FWD_EIS) num = (b0 - ua) - acc;
                    else if (MODE == SW_BWD_DIV) num = b0 - acc;
                    const R other = __shfl_xor_sync(0xffffffffu, num, 1);
                    // num.x and num.y as they meet lv.x and lv.y
                    R mine;
                    if (MODE == SW_BWD_IC) mine = cmadd(ua, lv, num, other);
                    else {
                        const T nm = im ? T{other, num} : T{num, other};
                        mine = cmul(nm, part(lv), im ? lv.x : lv.y);
                    }
                    wait_for(nd.z, nd.w);  // the own-ring slots are free
                    if (lead) ((R *)(X + ((h0.z + r) & (L.S_own - 1))))[im] = mine;
                    for (int k = 2; CL && k < hp.x; ++k)
                        if (lead) send(push[32 * k + r], mine, im * (int)sizeof(R));
                    __syncwarp();
                    if (lane == 0) tl_st_release(prog + 4u * warp, g + TS_W);
                    if (lead) {
                        send(to0, mine, im * (int)sizeof(R));
                        send(to1, mine, im * (int)sizeof(R));
                        tl_give((R *)(out + row) + im, mine);
                        if (MODE == SW_FWD_EIS) ((R *)(out2 + row))[im] = mine + ua;
                    }
                } else {
                    // Where the right-hand side is the larger part of the sum, every addition to it rounds at its size. The IC
                    // pair starts from it, as the push sweep did; the Eisenstat pair subtracted its lane sums last and takes
                    // it last here too, one multiply-add more behind the newest value (48^3 414 -> 439 us forward, 411 -> 417
                    // backward). Error of a sweep against long double, over the solution's norm, forward / backward, curl-curl
                    // 10^3 to 41^3: lane sums 0.91-0.98 / 0.93-0.98e-16, this 0.93-0.96 / 0.96-0.98e-16, starting from the
                    // right-hand side 1.18-1.27 / 1.25-1.34e-16; 5-point 100^2 0.74 / 0.76, 0.55 / 0.54, 0.81 / 0.82e-16.
                    constexpr bool late = MODE == SW_BWD_DIV || MODE == SW_FWD_EIS;
                    T res, u0 = Sc<T>::zero();
                    const int k1 = (h0.x >> 16) & 15, k2 = (h0.x >> 20) & 15;
                    lead = lane < cnt;  // lane r has row r outside the columns
                    // what the row starts from: on its way while the first block waits
                    T b0 = Sc<T>::zero(), lv = b0;
                    if (lead) {
                        if (CL && hp.x > 0) to0 = push[lane];
                        if (CL && hp.x > 1) to1 = push[32 + lane];
                        row = ((const int *)(rec + 16 * (of.w & 0xffff)))[lane];
                        if (MODE != SW_BWD_IC) {
                            lv = ((const T *)(rec + 16 * ((unsigned)of.w >> 16)))[lane];
                            b0 = rhs[row];
                        }
                        if (MODE == SW_BWD_IC || MODE == SW_FWD_EIS) u0 = aux[row];
                    }
                    // ---- columns: one or two lanes a row, the even and the odd columns in two sums
                    T s0 = Sc<T>::zero(), s1 = s0;
                    const ushort4 *c = (const ushort4 *)(rec + 16 * (of.y & 0xffff)) + lane;
                    int skip = 4 - h0.w;
#pragma unroll 1
                    for (int k = 0; k < nb; ++k) {
                        const int2 w = need[k];
                        const ushort4 cc = c[32 * k];
                        T vv[4], x0, x1, x2, x3;
                        tl_vals(v + 128 * k, lane, vv);
                        wait_for(w.x, w.y);
                        if (!cfar) {
                            x0 = X[cc.x], x1 = X[cc.y], x2 = X[cc.z], x3 = X[cc.w];
                        } else {
                            const int *f = cfar + 128 * k + 4 * lane;
                            x0 = value(cc.x, f), x1 = value(cc.y, f + 1), x2 = value(cc.z, f + 2), x3 = value(cc.w, f + 3);
                        }
                        // jumps, not predicates, past the first block's empty columns: a multiply-add costs the FP64
                        // latency whether or not it runs
                        if (lg) {
                            switch (skip) {
                                case 0: s0 = madd(s0, vv[0], x0); [[fallthrough]];
                                case 1: s0 = madd(s0, vv[1], x1); [[fallthrough]];
                                case 2: s0 = madd(s0, vv[2], x2); [[fallthrough]];
                                default: s0 = madd(s0, vv[3], x3);
                            }
                        } else {
                            switch (skip) {
                                case 0: s0 = madd(s0, vv[0], x0); [[fallthrough]];
                                case 1: s1 = madd(s1, vv[1], x1); [[fallthrough]];
                                case 2: s0 = madd(s0, vv[2], x2); [[fallthrough]];
                                default: s1 = madd(s1, vv[3], x3);
                            }
                        }
                        skip = 0;
                    }
                    if (nb > 0) {
                        if (lg) {
                            s0 = s0 + Sc<T>::shfl_xor(s0, 1);
                            s0 = Sc<T>::shfl(s0, (2 * lane) & 31);  // lane r takes row r's sum
                        } else {
                            s0 = s0 + s1;
                        }
                    }
                    if (MODE == SW_FWD_EIS) b0 = b0 - u0;
                    if (MODE == SW_BWD_IC) res = u0 + s0;
                    else res = late ? s0 : madd(s0, b0, lv);
                    // ---- tails: one lane a row; the first two values and codes of both stages ahead of the waits
                    const T *v1 = (const T *)(rec + 16 * ((unsigned)of.x >> 16)) + lane, *v2 = v1 + 32 * k1;
                    const unsigned short *c1 = (const unsigned short *)(rec + 16 * ((unsigned)of.y >> 16)) + lane,
                                         *c2 = c1 + 32 * k1;
                    // reads past a stage's entries stay inside the shared memory (tile_layout) and are not used
                    const T va = v1[0], vb = v1[32], wa = v2[0], wb = v2[32];
                    const int ca = c1[0], cb = c1[32], da = c2[0], db = c2[32];
                    if (k1 > 0) {
                        wait_for(nd.x, nd.y);
                        if (k1 > 1) {
                            const T xa = X[ca], xb = X[cb];
                            res = madd(res, va, xa);
                            res = madd(res, vb, xb);
#pragma unroll 1
                            for (int k = 2; k < k1; ++k) res = madd(res, v1[32 * k], X[c1[32 * k]]);
                        } else {
                            res = madd(res, va, X[ca]);
                        }
                    }
                    wait_for(nd.z, nd.w);
                    if (k2 > 0) {
                        if (k2 > 1) {
                            const T xa = X[da], xb = X[db];
                            res = madd(res, wa, xa);
                            res = madd(res, wb, xb);
#pragma unroll 1
                            for (int k = 2; k < k2; ++k) res = madd(res, v2[32 * k], X[c2[32 * k]]);
                        } else {
                            res = madd(res, wa, X[da]);
                        }
                    }
                    if (late) res = madd(res, b0, lv);
                    if (lead) X[(h0.z + lane) & (L.S_own - 1)] = res;
                    for (int k = 2; CL && k < hp.x; ++k)
                        if (lead) send(push[32 * k + lane], res, 0);
                    __syncwarp();
                    if (lane == 0) tl_st_release(prog + 4u * warp, g + TS_W);
                    if (lead) {
                        send(to0, res, 0);
                        send(to1, res, 0);
                        tl_give(out + row, res);
                        if (MODE == SW_FWD_EIS) out2[row] = res + u0;
                    }
                }
            }
        } else if (warp < TS_W + TS_R) {
            // ------------------------------------------------ receiver warps
            // chunk ch (32 values) is this warp's for ch % TS_R == me; a value counts as soon as it and all before it are here
            const int me = warp - TS_W;
            const unsigned count = prog + 4u * TS_W;
            const int *hl = a.halo + 32ll * td.z;
            int j = me < nch ? hl[32 * me + lane] : -1;
            int rel = me < nch ? a.rel[td.z + me] : -1;
            for (int ch = me; ch < nch; ch += TS_R) {
                const int jn = ch + TS_R < nch ? hl[32 * (ch + TS_R) + lane] : -1;
                const int reln = ch + TS_R < nch ? a.rel[td.z + ch + TS_R] : -1;
                // the slots' previous values are dead (they are, long since, unless the halo ring is full)
                if (rel >= 0) wait_for(rel, 0);
                bool have = j == -1, head = false;
                const bool pushed = CL && j == -2;
                T *const slot = X + L.S_own + ((32 * ch + lane) & (L.S_halo - 1));
                int told = 0, tries = 0;
                Bound b(a.err, lim);
                while (!bad) {
                    T x;
                    if (!have && (pushed ? tl_take(slot, x) : tl_take(out + j, x))) {
                        if (!pushed) *slot = x;
                        have = true;
                    }
                    const unsigned miss = ~__ballot_sync(0xffffffffu, have);
                    if (!head) head = __all_sync(0xffffffffu, tl_ld_acquire(count) >= 32 * ch);
                    const int now = miss ? __ffs(miss) - 1 : 32;
                    if (head && now > told) {
                        __syncwarp();
                        if (lane == 0) tl_st_release(count, 32 * ch + now);
                        told = now;
                    }
                    if (told == 32) break;
                    if (__any_sync(0xffffffffu, b.spent(63))) bad = true;
                    // far ahead of the producers: poll gently
                    if (++tries > 16 && __any_sync(0xffffffffu, !have && !pushed)) __nanosleep(100);
                }
                if (bad) break;
                j = jn;
                rel = reln;
            }
        } else {
            // ------------------------------------------------ staging warp
            for (int g0 = 0; g0 < ng && !bad; g0 += 32) {
                const int4 m = a.groups[td.x + min(g0 + lane, ng - 1)];
                for (int q = 0; q < 32 && g0 + q < ng; ++q) {
                    const int src = __shfl_sync(0xffffffffu, m.x, q), n16 = __shfl_sync(0xffffffffu, m.y, q);
                    const int dst = __shfl_sync(0xffffffffu, m.z, q), need = __shfl_sync(0xffffffffu, m.w, q);
                    if (need >= 0) wait_for(need, 0);
                    if (bad) break;
                    if (lane == 0) {
                        const unsigned bar = full + 8u * ((g0 + q) % TS_NM);
                        place[(g0 + q) % TS_NM] = dst;  // the arrival below releases it to the group's warp
                        tl_mbar_expect(bar, 16u * (unsigned)n16);
                        tl_bulk_g2s(sbase + L.o_rec + 16u * (unsigned)dst, a.rec + 16ll * src, 16u * (unsigned)n16, bar);
                    }
                    issued = g0 + q + 1;
                }
            }
        }
        if (__syncthreads_or(bad)) {
            // copies in flight land before the shared memory goes away (bounded)
            if (warp == TS_W + TS_R && lane == 0)
                for (int g = max(0, issued - TS_NM); g < issued; ++g) {
                    const unsigned long long t0 = gtimer();
                    while (!tl_mbar_test(full + 8u * (g % TS_NM), (unsigned)((g / TS_NM) & 1)) &&
                           gtimer() - t0 < 1000000ull) {
                    }
                }
            if (!CL) return;
            bad = true;  // the whole CTA goes on to the cluster's barriers and leaves with it
        }
        if (once) {
            if (CL) tl_cluster_sync();
            return;
        }
        if (tid < TS_NM) tl_mbar_inval(full + 8u * tid);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- record values (once per factor)
// by age rec[dval[k]] = -val[k] * lvec[t]; by lanes val[k], negated for the IC pair; rec[dlv[t]] = lvec[t]
enum : int { TF_SCALED = 0, TF_PLAIN = 1, TF_NEG = 2 };
template <typename T, int FILL>
__global__ void k_tile_fill(int n, const int *prp, const int *dval, const int *dlv, const T *val, const T *lvec, T *rec) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, q = threadIdx.x & 3;
    if (t >= n) return;
    const T lv = lvec[t];
    if (q == 0) rec[dlv[t]] = lv;
    for (int k = prp[t] + q; k < prp[t + 1]; k += 4) {
        const int d = dval[k];
        if (d >= 0) rec[d] = FILL == TF_SCALED ? -(val[k] * lv) : FILL == TF_NEG ? -val[k] : val[k];
    }
}

// the output vector unsolved, the ticket back at tile 0
template <typename W>
__global__ void k_tile_arm(W *p, size_t words, int *ticket, const KState *st) {
    if (st && !st->active) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x)
        p[i] = (W)~(W)0;
}

static int tile_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        sms = v > 0 ? v : 1;
    }
    return sms;
}

static TilePlan &tile_slot(Tri &T, int elem) { return T.tile[elem == 4 ? 0 : elem == 8 ? 1 : 2]; }

// another sweep serves the triangle; the buffers go back
static void tile_refuse(TilePlan &P) {
    for (DBuf *d : {&P.tiles, &P.groups, &P.halo, &P.rel, &P.dval, &P.dlv, &P.rec}) d->release();
    P.ready = false;
    P.failed = true;
}

// a triangle's pattern on the host
struct TilePattern {
    std::vector<int> prp, pci, ipos, level;
    void read(const Tri &T, cudaStream_t s) {
        const std::pair<std::vector<int> *, std::pair<const DBuf *, int>> arr[] = {
            {&prp, {&T.prp, T.n + 1}}, {&pci, {&T.pci, T.nnz}}, {&ipos, {&T.ipos, T.n}}, {&level, {&T.level, T.n}}};
        for (auto &a : arr) {
            a.first->resize((size_t)a.second.second);
            SSG_CUDA(cudaMemcpyAsync(a.first->data(), a.second.first->p, sizeof(int) * a.first->size(), cudaMemcpyDeviceToHost, s));
        }
    }
};

// false: no memory for it on the device
static bool tile_upload(TilePlan &P, const TilePlanHost &H, cudaStream_t s) {
    const std::pair<DBuf *, const std::vector<int> *> arr[] = {{&P.tiles, &H.tiles}, {&P.groups, &H.groups}, {&P.halo, &H.halo},
                                                               {&P.rel, &H.rel},     {&P.dval, &H.dval},     {&P.dlv, &H.dlv}};
    try {
        for (auto &a : arr) a.first->ensure(sizeof(int) * (a.second->size() + 4));
        P.rec.ensure((size_t)H.rec_bytes + 16);
    } catch (const Error &) {
        return false;
    }
    for (auto &a : arr)
        if (!a.second->empty())
            SSG_CUDA(cudaMemcpyAsync(a.first->p, a.second->data(), sizeof(int) * a.second->size(), cudaMemcpyHostToDevice, s));
    for (int t = 0; t < H.T; ++t)
        if (!H.rec[t].empty())
            SSG_CUDA(cudaMemcpyAsync(P.rec.as<unsigned char>() + H.rec_off[t], H.rec[t].data(), H.rec[t].size(),
                                     cudaMemcpyHostToDevice, s));
    SSG_CUDA(cudaStreamSynchronize(s));
    P.lay = H.lay;
    P.T = H.T;
    P.CS = H.CS;
    P.key_val = P.key_lv = nullptr;
    P.key_epoch = ~0ull;
    return true;
}

// The plans of a pair of triangles: once per pattern and value size, on the host (ss_tile_plan.cpp). A plan that does not
// fit, passes a limit or finds no memory, on the host or the device, is refused for good: the sync-free sweep, which needs
// none of it, then serves the pair.
bool tile_plan(Tri &a, Tri &b, size_t elem_bytes, int lanes, cudaStream_t s) {
    const int elem = (int)elem_bytes;
    bool all = true;
    for (Tri *T : {&a, &b}) {
        TilePlan &P = tile_slot(*T, elem);
        if (P.n != T->n || P.nnz != T->nnz || P.nlev != T->nlev || P.lanes != lanes) {
            P.ready = P.failed = false;
            P.lanes = lanes;
            P.n = T->n;
            P.nnz = T->nnz;
            P.nlev = T->nlev;
        }
        if (P.failed || T->n == 0) return false;
        all = all && P.ready;
    }
    if (all) return true;
    size_t here = 0, total = 0;
    SSG_CUDA(cudaMemGetInfo(&here, &total));
    const TileLimits lim = tile_limits(lanes, (long long)total);
    Tri *tri[2] = {&a, &b};
    TilePlanHost H[2];
    {
        TilePattern in[2];
        std::exception_ptr err[2];
        bool mine[2];  // to be planned
        for (int q = 0; q < 2; ++q) {
            mine[q] = !tile_slot(*tri[q], elem).ready;
            try {
                if (mine[q]) in[q].read(*tri[q], s);
            } catch (const std::bad_alloc &) {
                err[q] = std::current_exception();
            }
        }
        SSG_CUDA(cudaStreamSynchronize(s));
        auto plan = [&](int q) {
            const Tri &T = *tri[q];
            try {
                if (mine[q] && !err[q])
                    H[q] = tile_plan_host(T.n, T.nlev, in[q].prp.data(), in[q].pci.data(), in[q].ipos.data(), in[q].level.data(),
                                          T.lower, elem, lanes, 0, tile_cluster(tile_count(T.n, lanes), lanes), nullptr, &lim);
            } catch (...) {
                err[q] = std::current_exception();
            }
        };
        // both at a time (80^3: 407 ms one after the other, 180 with the last pass on all threads and side by side)
        std::thread other;
        try {
            if (mine[0] && mine[1]) other = std::thread(plan, 1);
        } catch (...) {
        }
        plan(0);
        if (other.joinable()) other.join();
        else plan(1);
        for (int q = 0; q < 2; ++q) {
            try {
                if (err[q]) std::rethrow_exception(err[q]);
            } catch (const std::bad_alloc &) {
            }
            if (mine[q] && !H[q].ok) {
                tile_refuse(tile_slot(*tri[q], elem));
                return false;
            }
        }
    }
    for (int q = 0; q < 2; ++q) {
        TilePlan &P = tile_slot(*tri[q], elem);
        if (P.ready) continue;
        if (!tile_upload(P, H[q], s)) {
            tile_refuse(P);
            // the other one is of no use without it
            if (q == 1 && H[0].ok) {
                tile_refuse(tile_slot(a, elem));
                tile_slot(a, elem).failed = false;
            }
            return false;
        }
        P.ready = true;
    }
    return true;
}

template <typename T>
void sweep_tile(Tri &tri, const T *val, int mode, const T *rhs, const T *aux, const T *lvec, unsigned long long epoch,
                T *out, T *out2, int *ticket, const KState *st, int *err, cudaStream_t s) {
    TilePlan &P = tile_slot(tri, (int)sizeof(T));
    if (tri.n == 0) return;
    if (!P.ready || P.n != tri.n || P.nnz != tri.nnz || P.nlev != tri.nlev)
        throw Error{SSG_ERR_STATE, "tile sweep without a plan for this triangle"};
    constexpr bool by_lanes = Sc<T>::is_complex;
    const int fill = !by_lanes ? TF_SCALED : mode == SW_FWD_DIV || mode == SW_BWD_IC ? TF_NEG : TF_PLAIN;
    if (P.key_val != val || P.key_lv != lvec || P.key_epoch != epoch || P.key_fill != fill) {
        auto k = fill == TF_SCALED ? k_tile_fill<T, TF_SCALED> : fill == TF_NEG ? k_tile_fill<T, TF_NEG> : k_tile_fill<T, TF_PLAIN>;
        k<<<div_up((long long)tri.n * 4, 256), 256, 0, s>>>(tri.n, tri.prp.as<int>(), P.dval.as<int>(), P.dlv.as<int>(), val,
                                                            lvec, P.rec.as<T>());
        SSG_LAUNCHED();
        P.key_val = val;
        P.key_lv = lvec;
        P.key_epoch = epoch;
        P.key_fill = fill;
    }
    {
        using W = unsigned long long;
        const size_t bytes = sizeof(T) * (size_t)tri.n;
        if (bytes % 8 == 0 && ((size_t)out & 7) == 0)
            k_tile_arm<W><<<std::min(div_up((long long)(bytes / 8), 1024), 4 * tile_sms()), 256, 0, s>>>(
                (W *)out, bytes / 8, ticket, st);
        else
            k_tile_arm<unsigned><<<std::min(div_up((long long)(bytes / 4), 1024), 4 * tile_sms()), 256, 0, s>>>(
                (unsigned *)out, bytes / 4, ticket, st);
        SSG_LAUNCHED();
    }
    TileArgs a;
    a.T = P.T;
    a.CS = P.CS;
    a.tiles = P.tiles.as<int4>();
    a.groups = P.groups.as<int4>();
    a.halo = P.halo.as<int>();
    a.rel = P.rel.as<int>();
    a.rec = P.rec.as<unsigned char>();
    a.rhs = rhs;
    a.aux = aux;
    a.out = out;
    a.out2 = out2;
    a.ticket = ticket;
    a.st = st;
    a.err = err;
    a.L = P.lay;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = P.CS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(TS_THREADS);
    cfg.dynamicSmemBytes = P.lay.total;
    cfg.stream = s;
    cfg.gridDim = dim3(std::min((P.T + P.CS - 1) / P.CS, std::max(1, tile_sms() / P.CS)) * P.CS);
#define SSG_TS(M, LN, CL)                                                                                      \
    do {                                                                                                       \
        auto kern = k_sweep_tile<T, M, LN, CL>;                                                                \
        static bool prepared = false;                                                                          \
        if (!prepared) {                                                                                       \
            SSG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX));    \
            prepared = true;                                                                                   \
        }                                                                                                      \
        SSG_CUDA(cudaLaunchKernelEx(&cfg, kern, a));                                                           \
    } while (0)
#define SSG_TM(LN, CL)                                                     \
    switch (mode) {                                                        \
        case SW_FWD_DIV: SSG_TS(SW_FWD_DIV, LN, CL); break;                \
        case SW_BWD_IC: SSG_TS(SW_BWD_IC, LN, CL); break;                  \
        case SW_BWD_DIV: SSG_TS(SW_BWD_DIV, LN, CL); break;                \
        default: SSG_TS(SW_FWD_EIS, LN, CL); break;                        \
    }
    if constexpr (!by_lanes) {
        if (P.CS > 1) {
            SSG_TM(0, true)
        } else {
            SSG_TM(0, false)
        }
    } else if (P.lanes == 4) {
        SSG_TM(4, false)
    } else {
        SSG_TM(8, false)
    }
#undef SSG_TM
#undef SSG_TS
    SSG_LAUNCHED();
}

#define SSG_INST(T)                                                                                              \
    template void sweep_tile<T>(Tri &, const T *, int, const T *, const T *, const T *, unsigned long long, T *, \
                                T *, int *, const KState *, int *, cudaStream_t);
SSG_INST(double)
SSG_INST(cplx)
SSG_INST(float)
SSG_INST(cplxf)
#undef SSG_INST

}  // namespace ssg
