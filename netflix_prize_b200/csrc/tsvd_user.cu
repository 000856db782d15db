// User stratum of the stratified schedule without the per-day terms
// (fit_epoch_user, src/tsvdx4p.rs:390-639): users in parallel, item tables
// frozen, one warp per user, the user's ratings in order, two at a time.
//
// The item rows qe_k = q_i + q^f_{i,0} do not change in this stratum, and every
// update is affine in the user's state, so the second rating's error follows
// from the state before the first:
//   err_0 = C_0,  err_1 = C_1 - M err_0,
// C_k from the state at the pair's start (with the decay of the rating before
// it), M the effect of err_0 on rating 1 through p_u, p2_u, the biases, alpha_u,
// the day's bias and c_u. One reduction of three sums (two dots and qe_0 . qe_1)
// replaces two dependent ones, and the rows are read and scaled once per pair.
//
// Larger blocks cost no fewer instructions per rating and lose more than they
// save: a loop of about 180 instructions stays in the instruction cache next to
// the schedulers, one of 500 (blocks of four) waited 3.5 cycles for every
// instruction it issued.
//
// The rows come through a ring of shared-memory slots per warp, asked for
// kAheadRows ratings ahead, so their latency takes no registers.
//
// Bound by issue and the fixed latencies of the pair's chain; the rows (1 KB a
// rating at f = 256) come from L2, which holds the table. Measured against one
// rating at a time (one B200, CUDA events): 100,480,507 ratings, f = 256, 24.2 ->
// 16.0 ms; 25 M ratings, f = 64, 9.2 -> 3.5 ms; 1 M ratings, f = 32, 0.74 ->
// 0.45 ms.
#include <algorithm>

#include "tsvd_chain.cuh"

namespace tsvd {
namespace {

constexpr int kUThreads = 128;
constexpr int kRingRows = 8;    // slots of a warp's ring
constexpr int kAheadRows = 6;   // ratings asked for ahead (even, < kRingRows - 1)

// CTAs per SM the registers are bounded for: the most that spill nothing (at f =
// 256 one more CTA, with 56 bytes spilled, measured 17.5 against 16.0 ms).
constexpr int user_ctas(int vpl) { return vpl >= 7 ? 4 : vpl >= 5 ? 5 : vpl >= 3 ? 6 : 7; }

template <int VPL, bool ORD>
__global__ void __launch_bounds__(kUThreads, user_ctas(VPL)) k_user_pairs(DeviceState s, EpochParams p, Bf16Copies bf,
                                                                          const uint32_t* __restrict__ order,
                                                                          uint32_t n_work) {
    using V = Vec<VPL>;
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF;
    float* ring = smem + (threadIdx.x >> 5) * kRingRows * Fs;
    float th[4];
    if constexpr (ORD) load_thresholds(s, th);
    // x - lr (g + reg x) = x + (a - 1) x - lr g, a = 1 - lr reg; c_u decays towards
    // 1. A row's decay is added as (a - 1) x: multiplying by a rounded to FP32
    // would be off by the same factor at every rating.
    const float da = -p.lr_u * p.reg_u, db = -p.lr_u2 * p.reg_u2, dc = -p.lr_cu * p.reg_cu;
    const float a1 = 1.0f + da, b1 = 1.0f + db, c1 = 1.0f + dc;
    const float da2 = fmaf(da, da, 2.0f * da), db2 = fmaf(db, db, 2.0f * db), dc2 = fmaf(dc, dc, 2.0f * dc);
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&s.counters[0], 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= n_work) break;
        const uint32_t u = order[k];
        const uint64_t start = s.user_off[u], end = s.user_off[u + 1];
        if (start == end) continue;
        const uint64_t ps = s.pr_off[u], pe = s.pr_off[u + 1];
        const uint64_t total = (end - start) + (p.full_su ? (pe - ps) : 0);
        const float norm = sqrtf((float)total);

        // su (src/tsvdx4p.rs:466-491): equals ycache[u] bit for bit when full_su
        // holds and ycache was rebuilt from the current y.
        V su;
        float sub;
        if (p.use_ycache) {
            su.load_cg(s.ycache + (size_t)u * Fs, lane);
            sub = __ldcg(s.ycache_bias + u);
        } else {
            su.zero();
            sub = 0.0f;
            const Rec* rr = s.rec + start;
            const uint32_t* pp = s.pr_item + ps;
            auto train = [&](uint64_t q) { return rec_id(__ldg(&rr[q].key)); };
            auto probe = [&](uint64_t q) { return __ldg(pp + q); };
            const uint64_t n_pr = p.full_su ? pe - ps : 0;
            if (bf.yfeat) {
                sum_rows<VPL, true>(nullptr, bf.yfeat, s.ybias, Fs, end - start, train, lane, su, sub);
                sum_rows<VPL, true>(nullptr, bf.yfeat, s.ybias, Fs, n_pr, probe, lane, su, sub);
            } else {
                sum_rows<VPL, false>(s.yfeat, nullptr, s.ybias, Fs, end - start, train, lane, su, sub);
                sum_rows<VPL, false>(s.yfeat, nullptr, s.ybias, Fs, n_pr, probe, lane, su, sub);
            }
            su.divide(norm);
            sub = sub / norm;
            su.store_cg(s.ycache + (size_t)u * Fs, lane);
            if (lane == 0) s.ycache_bias[u] = sub;
        }

        V pu, p2, seq;
        pu.load_cg(s.ufeat + (size_t)u * Fs, lane);
        p2.load_cg(s.ufeat2 + (size_t)u * Fs, lane);
        seq.zero();
        float ub = __ldcg(s.ubias + u), al = __ldcg(s.alpha_u + u);
        float cm = __ldcg(s.cu + u) - 1.0f;  // c_u - 1
        float bb0 = lane < (int)T ? __ldcg(s.but_bin + (size_t)u * T + lane) : 0.0f;
        float bb1 = lane + 32 < (int)T ? __ldcg(s.but_bin + (size_t)u * T + 32 + lane) : 0.0f;
        float sum_err = 0.0f;

        // a chunk's records, one rating per lane, a chunk ahead; lanes past the end
        // take the last rating (its loads are valid, its weight zero)
        auto chunk_rec = [&](uint64_t base) { return load_rec(s.rec + min(base + lane, end - 1)); };
        Rec ahead = chunk_rec(start);
        // rating j of the chunk whose keys are `keys` into slot j % kRingRows
        auto ask = [&](uint32_t keys, uint32_t j) {
            const uint32_t i = rec_id(__shfl_sync(kFull, keys, j));
            row_cp_async<VPL>(ring + (j % kRingRows) * Fs, s.qe0 + (size_t)i * Fs, lane);
        };
#pragma unroll
        for (int q = 0; q < kAheadRows; q += 2) {
            ask(ahead.key, q);
            ask(ahead.key, q + 1);
            cp_async_commit();
        }
        for (uint64_t base = start; base < end; base += 32) {
            const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
            const Rec r = ahead;
            ahead = chunk_rec(base + 32);
            const uint32_t i = rec_id(r.key), tb = rec_tbin(r.key);
            const bool hud = r.ud < s.n_ud;
            // low_memory: training uses frequency bin 0 (src/tsvdx4p.rs:504-531)
            const float bi = __ldg(s.ibias + i) + __ldg(s.bit_bin + (size_t)i * T + tb) + __ldg(s.ibias_freq + (size_t)i * NF);
            const float ct = hud ? __ldg(s.cut + r.ud) : 0.0f;
            // the day's and the time bin's bias, kept current for every rating of the chunk
            float bud = hud ? __ldcg(s.ubias_day + r.ud) : 0.0f, but;
            {
                const float t0 = __shfl_sync(kFull, bb0, tb & 31), t1 = __shfl_sync(kFull, bb1, tb & 31);
                but = tb < 32 ? t0 : t1;
            }
            const float c0 = s.gbias + sub + bi * (1.0f + ct) - (ORD ? 0.0f : r.res);
            // M's parts for this lane's rating and the next one's: M = mb + mg qe_0 . qe_1
            float mb, mg;
            {
                const float dn = __shfl_down_sync(kFull, r.dev, 1), bn = __shfl_down_sync(kFull, bi, 1);
                const uint32_t un = __shfl_down_sync(kFull, r.ud, 1), tn = __shfl_down_sync(kFull, tb, 1);
                const float dd = r.dev * dn;
                mb = p.lr_ub + p.lr_ta * dd + (tn == tb ? p.lr_tu : 0.0f) + (hud && un == r.ud ? p.lr_ubd : 0.0f) +
                     p.lr_cu * (bi * bn);
                mg = p.lr_u + p.lr_u2 * dd;
            }
#pragma unroll 1
            for (uint32_t j = 0; j < cnt; j += 2) {
                {  // two rows more, of the next chunk where this one ends
                    const bool here = j + kAheadRows < 32;
                    const uint32_t keys = here ? r.key : ahead.key, q = (j + kAheadRows) & 31u;
                    ask(keys, q);
                    ask(keys, q + 1);
                    cp_async_commit();
                }
                cp_async_wait<kAheadRows / 2>();
                V q0, q1;
                q0.load(ring + (j % kRingRows) * Fs, lane);
                q1.load(ring + ((j + 1) % kRingRows) * Fs, lane);
                const bool two = j + 1 < cnt;
                const float d0 = __shfl_sync(kFull, r.dev, j), d1 = __shfl_sync(kFull, r.dev, j + 1);
                float v0, v1, g = q0.dot(q1);
                {
                    V t = su;
                    t.fma(d0, p2);
                    t.add(pu);
                    v0 = q0.dot(t);
                    t = su;
                    t.fma(b1 * d1, p2);
                    t.fma(a1, pu);
                    v1 = q1.dot(t);
                }
                // the three sums: (v0 | v1) and g, then (v | g)
                {
                    const bool up = (lane & 16) != 0;
                    const float keep = up ? v1 : v0, send = up ? v0 : v1;
                    v0 = keep + __shfl_xor_sync(kFull, send, 16);
                    g += __shfl_xor_sync(kFull, g, 16);
                    const bool up8 = (lane & 8) != 0;
                    const float keep8 = up8 ? g : v0, send8 = up8 ? v0 : g;
                    v0 = keep8 + __shfl_xor_sync(kFull, send8, 8);
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) v0 += __shfl_xor_sync(kFull, v0, o);
                    v1 = __shfl_sync(kFull, v0, 16);
                    g = __shfl_sync(kFull, v0, 8);
                    v0 = __shfl_sync(kFull, v0, 0);
                }
                const float cl = c0 + but + bud;
                const float bi0 = __shfl_sync(kFull, bi, j), bi1 = __shfl_sync(kFull, bi, j + 1);
                float e0 = __shfl_sync(kFull, cl, j) + ub + al * d0 + bi0 * cm + v0;
                float e1 = __shfl_sync(kFull, cl, j + 1) + ub + al * d1 + bi1 * (c1 * cm) + v1;
                const float m10 = __shfl_sync(kFull, mb, j) + __shfl_sync(kFull, mg, j) * g;
                if constexpr (ORD) e0 = ordinal_grad(th, e0, (int)__shfl_sync(kFull, r.res, j));
                e1 = fmaf(-m10, e0, e1);
                if constexpr (ORD) e1 = ordinal_grad(th, e1, (int)__shfl_sync(kFull, r.res, j + 1));
                // a last rating without a second: no update and no decay from it
                e1 = two ? e1 : 0.0f;
                const float a2 = two ? a1 : 1.0f, b2 = two ? b1 : 1.0f, c2 = two ? c1 : 1.0f;
                seq.fma(e0, q0);
                seq.fma(e1, q1);
                // each row's change is summed first and rounded into the row once
                V t = pu;
                t.scale(two ? da2 : da);
                t.fma(-p.lr_u * a2 * e0, q0);
                t.fma(-p.lr_u * e1, q1);
                pu.add(t);
                t = p2;
                t.scale(two ? db2 : db);
                t.fma(-p.lr_u2 * b2 * (e0 * d0), q0);
                t.fma(-p.lr_u2 * (e1 * d1), q1);
                p2.add(t);
                sum_err += e0;
                sum_err += e1;
                ub -= p.lr_ub * (e0 + e1);
                al -= p.lr_ta * fmaf(e0, d0, e1 * d1);
                cm = fmaf(two ? dc2 : dc, cm, cm) - p.lr_cu * fmaf(c2 * e0, bi0, e1 * bi1);
                {
                    const uint32_t u0 = __shfl_sync(kFull, r.ud, j), u1 = __shfl_sync(kFull, r.ud, j + 1);
                    const float w0 = hud && u0 == r.ud ? e0 : 0.0f, w1 = hud && u1 == r.ud ? e1 : 0.0f;
                    bud -= p.lr_ubd * (w0 + w1);
                }
                if (p.lr_tu != 0.0f) {
                    const uint32_t t0 = __shfl_sync(kFull, tb, j), t1 = __shfl_sync(kFull, tb, j + 1);
                    but -= p.lr_tu * ((t0 == tb ? e0 : 0.0f) + (t1 == tb ? e1 : 0.0f));
                    const uint32_t lo = lane, hi = lane + 32;
                    bb0 -= p.lr_tu * ((t0 == lo ? e0 : 0.0f) + (t1 == lo ? e1 : 0.0f));
                    bb1 -= p.lr_tu * ((t0 == hi ? e0 : 0.0f) + (t1 == hi ? e1 : 0.0f));
                }
            }
            // the chunk's day biases (ratings of one day hold the same value)
            if (hud) __stcg(s.ubias_day + r.ud, bud);
            __syncwarp();
        }
        cp_async_wait<0>();
        pu.store_cg(s.ufeat + (size_t)u * Fs, lane);
        p2.store_cg(s.ufeat2 + (size_t)u * Fs, lane);
        if (lane == 0) {
            s.ubias[u] = ub;
            s.alpha_u[u] = al;
            s.cu[u] = cm + 1.0f;
        }
        if (lane < (int)T) s.but_bin[(size_t)u * T + lane] = bb0;
        if (lane + 32 < (int)T) s.but_bin[(size_t)u * T + 32 + lane] = bb1;
        seq.divide(norm);
        seq.store_cg(s.g_user + (size_t)u * Fs, lane);
        if (lane == 0) s.e_user[u] = sum_err / norm;
    }
}

template <int VPL, bool ORD>
void launch_user(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf, const uint32_t* work,
                 uint32_t n) {
    auto kern = k_user_pairs<VPL, ORD>;
    const size_t smem = (size_t)(kUThreads / 32) * kRingRows * s.Fs * sizeof(float);
    int dev = 0, sms = 0, per_sm = 0;
    TSVD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TSVD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kUThreads, smem));
    kern<<<(unsigned)(sms * std::max(per_sm, 1)), kUThreads, smem, m->stream>>>(s, p, bf, work, n);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

// ---------------------------------------------------------------------------
// With the per-day terms (low_memory = false): one rating at a time. Each run of
// equal dates gets its su_day from yfeat_day (the run's training items, then the
// day's pr items, src/tsvdx4p.rs:500-527), the ratings add ufeat_day and su_day to
// p_u(t), ufeat_day is trained (:604-611), and at the run's end its error sum over
// sqrt(day count) goes to every item of the run as a yfeat_day delta (:614-622).
//
// A run is a rating or two, so what it starts with decides the chain: its
// ufeat_day row and its first yfeat_day row are asked for while the run before it
// is trained (the two runs' days differ, so the row is not about to change), its
// length comes from the chunk's records in registers, and the item rows come
// through the ring. 6 M ratings, f = 60: 17.9 ms when each of these was waited for
// in turn, DAYMS now.
// ---------------------------------------------------------------------------
constexpr int day_ctas(int vpl) { return vpl >= 7 ? 3 : vpl >= 5 ? 4 : vpl >= 3 ? 5 : 7; }

// Fixed-point accumulation of a per-day NSVD1 delta row (red.global.add.u64).
template <int VPL>
__device__ __forceinline__ void dyd_add(unsigned long long* row, int lane, const float (&x)[VPL]) {
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        const long long q = __double2ll_rn((double)x[v] * kDydScale);
        atomicAdd(row + Row<VPL>::elem(lane, v), (unsigned long long)q);
    }
}

template <int VPL>
__global__ void __launch_bounds__(kUThreads, day_ctas(VPL)) k_user_days(DeviceState s, EpochParams p,
                                                                        const uint32_t* __restrict__ order,
                                                                        uint32_t n_work) {
    using V = Vec<VPL>;
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF;
    float* ring = smem + (threadIdx.x >> 5) * kRingRows * 2 * Fs;
    const bool ordinal = s.raw != nullptr;
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&s.counters[0], 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= n_work) break;
        const uint32_t u = order[k];
        const uint64_t start = s.user_off[u], end = s.user_off[u + 1];
        if (start == end) continue;
        const uint64_t ps = s.pr_off[u], pe = s.pr_off[u + 1];
        const uint64_t total = (end - start) + (p.full_su ? (pe - ps) : 0);
        const float norm = sqrtf((float)total);
        V su;
        float sub;
        if (p.use_ycache) {
            su.load_cg(s.ycache + (size_t)u * Fs, lane);
            sub = __ldcg(s.ycache_bias + u);
        } else {
            su.zero();
            sub = 0.0f;
            const Rec* rr = s.rec + start;
            const uint32_t* pp = s.pr_item + ps;
            sum_rows<VPL, false>(s.yfeat, nullptr, s.ybias, Fs, end - start,
                                 [&](uint64_t q) { return rec_id(__ldg(&rr[q].key)); }, lane, su, sub);
            sum_rows<VPL, false>(s.yfeat, nullptr, s.ybias, Fs, p.full_su ? pe - ps : 0,
                                 [&](uint64_t q) { return __ldg(pp + q); }, lane, su, sub);
            su.divide(norm);
            sub = sub / norm;
            su.store_cg(s.ycache + (size_t)u * Fs, lane);
            if (lane == 0) s.ycache_bias[u] = sub;
        }
        V pu, p2, seq;
        pu.load_cg(s.ufeat + (size_t)u * Fs, lane);
        p2.load_cg(s.ufeat2 + (size_t)u * Fs, lane);
        seq.zero();
        float ub = __ldcg(s.ubias + u), al = __ldcg(s.alpha_u + u), cuu = __ldcg(s.cu + u);
        float bb0 = lane < (int)T ? __ldcg(s.but_bin + (size_t)u * T + lane) : 0.0f;
        float bb1 = lane + 32 < (int)T ? __ldcg(s.but_bin + (size_t)u * T + 32 + lane) : 0.0f;
        float sum_err = 0.0f;
        // the current run of equal dates, and the next one's first rows
        V sud, seqd, pud, sn, pn;
        float norm_day = 1.0f;
        uint64_t run0 = 0, run1 = 0;

        auto chunk_rec = [&](uint64_t base) { return load_rec(s.rec + min(base + lane, end - 1)); };
        Rec ahead = chunk_rec(start);
        // rating j of the chunk whose keys are `keys`: its item's q and q^f row
        auto ask = [&](uint32_t keys, uint32_t j) {
            const uint32_t key = __shfl_sync(kFull, keys, j);
            float* slot = ring + (j % kRingRows) * 2 * Fs;
            row_cp_async<VPL>(slot, s.ifeat + (size_t)rec_id(key) * Fs, lane);
            row_cp_async<VPL>(slot + Fs, s.ifeat_freq + ((size_t)rec_id(key) * NF + rec_fbin(key)) * Fs, lane);
            cp_async_commit();
        };
        auto ask_run = [&](uint32_t key, uint32_t ud) {
            if (p.has_ud && ud < s.n_ud) pn.load_cg(s.ufeat_day + (size_t)ud * Fs, lane);
            else pn.zero();
            sn.load_nc(s.yfeat_day + (size_t)rec_id(key) * Fs, lane);
        };
#pragma unroll 1
        for (int q = 0; q < kAheadRows; ++q) ask(ahead.key, q);
        ask_run(__shfl_sync(kFull, ahead.key, 0), __shfl_sync(kFull, ahead.ud, 0));
        for (uint64_t base = start; base < end; base += 32) {
            const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
            const Rec r = ahead;
            ahead = chunk_rec(base + 32);
            const uint32_t i = rec_id(r.key), tb = rec_tbin(r.key);
            const bool hud = r.ud < s.n_ud;
            const float bi = __ldg(s.ibias + i) + __ldg(s.bit_bin + (size_t)i * T + tb) +
                             __ldg(s.ibias_freq + (size_t)i * NF + rec_fbin(r.key));
            const float ct = hud ? __ldg(s.cut + r.ud) : 0.0f;
            const uint32_t pr_day = p.full_su && hud ? __ldg(s.ud_pr_cnt + r.ud) : 0u;
            // the day's bias, kept current for every rating of the chunk
            float bud = hud ? __ldcg(s.ubias_day + r.ud) : 0.0f;
            // lanes whose rating ends a run (the chunk's last: by the next chunk's first)
            uint32_t un = __shfl_down_sync(kFull, r.ud, 1);
            const uint32_t u_next = __shfl_sync(kFull, ahead.ud, 0);
            if (lane == 31) un = u_next;
            const unsigned ends = __ballot_sync(kFull, un != r.ud || base + lane + 1 >= end);
#pragma unroll 1
            for (uint32_t j = 0; j < cnt; ++j) {
                {
                    const bool here = j + kAheadRows < 32;
                    ask(here ? r.key : ahead.key, (j + kAheadRows) & 31u);
                }
                const uint64_t t = base + j;
                const uint32_t uj = __shfl_sync(kFull, r.ud, j), kj = __shfl_sync(kFull, r.key, j);
                const bool hj = uj < s.n_ud;
                if (t == start || t > run1) {
                    // a new run of equal dates (day_ranges, src/tx.rs:92-104)
                    const unsigned later = ends & ~((1u << j) - 1u);
                    run1 = later ? base + __ffs((int)later) - 1 : base + 31;
                    if (!later)
                        while (run1 + 1 < end && __ldg(&s.rec[run1 + 1].ud) == uj) ++run1;
                    run0 = t;
                    pud = pn;
                    sud = sn;
                    seqd.zero();
                    const uint32_t pc = __shfl_sync(kFull, pr_day, j);
                    const float day_cnt = (float)(uint32_t)(run1 - t + 1) + (float)pc;
                    float none = 0.0f;
                    if (run1 > t)
                        sum_rows<VPL, false>(s.yfeat_day, nullptr, nullptr, Fs, run1 - t,
                                             [&](uint64_t q) { return rec_id(__ldg(&s.rec[t + 1 + q].key)); }, lane, sud,
                                             none);
                    if (pc) {
                        const uint32_t* list = s.ud_list_item + s.ud_list_off[uj];
                        sum_rows<VPL, false>(s.yfeat_day, nullptr, nullptr, Fs, pc,
                                             [&](uint64_t q) { return __ldg(list + q); }, lane, sud, none);
                    }
                    norm_day = sqrtf(day_cnt);
                    if (day_cnt != 1.0f) sud.divide(norm_day);
                    const uint64_t nr = run1 + 1;
                    if (nr < end) {
                        const uint32_t at = (uint32_t)(nr - base);
                        if (at < 64) {
                            const uint32_t nk = __shfl_sync(kFull, at < 32 ? r.key : ahead.key, at & 31);
                            ask_run(nk, __shfl_sync(kFull, at < 32 ? r.ud : ahead.ud, at & 31));
                        } else {
                            const Rec n = load_rec(s.rec + nr);
                            ask_run(n.key, n.ud);
                        }
                    }
                }
                cp_async_wait<kAheadRows>();
                V qe;
                {
                    V f;
                    const float* slot = ring + (j % kRingRows) * 2 * Fs;
                    qe.load(slot, lane);
                    f.load(slot + Fs, lane);
                    qe.add(f);  // q_i + q^f_{i,fb}
                }
                const float dv = __shfl_sync(kFull, r.dev, j);
                float dot;
                {
                    V x = su;
                    x.add(pu);
                    x.fma(dv, p2);
                    x.add(pud);
                    x.add(sud);
                    dot = warp_sum(qe.dot(x));
                }
                const uint32_t tj = rec_tbin(kj);
                const float but = __shfl_sync(kFull, tj < 32 ? bb0 : bb1, tj & 31);
                const float bi_t = __shfl_sync(kFull, bi, j);
                const float bu_t = ub + but + al * dv + __shfl_sync(kFull, bud, j) + sub;
                const float score = s.gbias + bu_t + bi_t * (cuu + __shfl_sync(kFull, ct, j)) + dot;
                const float target = __shfl_sync(kFull, r.res, j);
                const float err = ordinal ? ordinal_err(s.thresholds, score, (int)target) : score - target;
                ub -= p.lr_ub * err;
                {
                    const float nb = but - p.lr_tu * err;
                    if (lane == (int)(tj & 31)) {
                        if (tj < 32) bb0 = nb;
                        else bb1 = nb;
                    }
                }
                al -= p.lr_ta * err * dv;
                bud -= hud && uj == r.ud ? p.lr_ubd * err : 0.0f;
                cuu -= p.lr_cu * (err * bi_t + p.reg_cu * (cuu - 1.0f));
                sum_err += err;
                seq.fma(err, qe);
                seqd.fma(err, qe);
                // x - lr (g + reg x), the change rounded into the row once
                {
                    V x = pu;
                    x.scale(-p.lr_u * p.reg_u);
                    x.fma(-p.lr_u * err, qe);
                    pu.add(x);
                    x = p2;
                    x.scale(-p.lr_u2 * p.reg_u2);
                    x.fma(-p.lr_u2 * (err * dv), qe);
                    p2.add(x);
                    if (p.has_ud && hj) {
                        x = pud;
                        x.scale(-p.lr_ud * p.reg_ud);
                        x.fma(-p.lr_ud * err, qe);
                        pud.add(x);
                    }
                }
                if (t == run1) {
                    // end of the run: ufeat_day back, and the run's yfeat_day delta to
                    // each of its items
                    if (p.has_ud && hj) pud.store_cg(s.ufeat_day + (size_t)uj * Fs, lane);
                    seqd.divide(norm_day);
                    float gd[VPL];
                    seqd.to(gd);
                    dyd_add<VPL>(s.dyd_fix + (size_t)rec_id(kj) * Fs, lane, gd);
                    for (uint64_t q = run0; q < run1; ++q)
                        dyd_add<VPL>(s.dyd_fix + (size_t)rec_id(__ldg(&s.rec[q].key)) * Fs, lane, gd);
                }
            }
            // the chunk's day biases (ratings of one day hold the same value)
            if (hud) __stcg(s.ubias_day + r.ud, bud);
            __syncwarp();
        }
        cp_async_wait<0>();
        pu.store_cg(s.ufeat + (size_t)u * Fs, lane);
        p2.store_cg(s.ufeat2 + (size_t)u * Fs, lane);
        if (lane == 0) {
            s.ubias[u] = ub;
            s.alpha_u[u] = al;
            s.cu[u] = cuu;
        }
        if (lane < (int)T) s.but_bin[(size_t)u * T + lane] = bb0;
        if (lane + 32 < (int)T) s.but_bin[(size_t)u * T + 32 + lane] = bb1;
        seq.divide(norm);
        seq.store_cg(s.g_user + (size_t)u * Fs, lane);
        if (lane == 0) s.e_user[u] = sum_err / norm;
    }
}

template <int VPL>
void launch_days(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n) {
    auto kern = k_user_days<VPL>;
    const size_t smem = (size_t)(kUThreads / 32) * kRingRows * 2 * s.Fs * sizeof(float);
    int dev = 0, sms = 0, per_sm = 0;
    TSVD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TSVD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kUThreads, smem));
    kern<<<(unsigned)(sms * std::max(per_sm, 1)), kUThreads, smem, m->stream>>>(s, p, work, n);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

}  // namespace

void launch_user_stratum(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf,
                         const uint32_t* work, uint32_t n) {
    const int vpl = (int)(s.Fs / 32);
    if (s.raw) {
        TSVD_DISPATCH(vpl, (launch_user<V, true>(m, s, p, bf, work, n)));
    } else {
        TSVD_DISPATCH(vpl, (launch_user<V, false>(m, s, p, bf, work, n)));
    }
}

void launch_user_days(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n) {
    TSVD_DISPATCH((int)(s.Fs / 32), launch_days<V>(m, s, p, work, n));
}

}  // namespace tsvd
