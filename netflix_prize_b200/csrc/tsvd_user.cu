// User stratum of the stratified schedule, rows up to 256 columns (fit_epoch_user,
// src/tsvdx4p.rs:390-639): users in parallel, item tables frozen, one warp per user,
// the user's ratings in order, two at a time.
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
// Larger blocks cost no fewer instructions per rating and a longer loop: blocks of
// four took 26.8 ms at 100,480,507 ratings, f = 256, where pairs take 16.0.
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

// su (src/tsvdx4p.rs:466-491): equals ycache[u] bit for bit when full_su holds and
// ycache was rebuilt from the current y.
template <int VPL>
__device__ __forceinline__ void load_su(const DeviceState& s, const EpochParams& p, const Bf16Copies& bf, uint32_t u,
                                        uint64_t start, uint64_t end, float norm, int lane, Vec<VPL>& su, float& sub) {
    if (p.use_ycache) {
        su.load_cg(s.ycache + (size_t)u * s.Fs, lane);
        sub = __ldcg(s.ycache_bias + u);
        return;
    }
    const uint32_t Fs = s.Fs;
    const uint64_t ps = s.pr_off[u], pe = s.pr_off[u + 1];
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

        V su;
        float sub;
        load_su<VPL>(s, p, bf, u, start, end, norm, lane, su, sub);

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
    allow_dyn_smem(kern, smem);
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TSVD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kUThreads, smem));
    kern<<<(unsigned)(sms * std::max(per_sm, 1)), kUThreads, smem, m->stream>>>(s, p, bf, work, n);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

// ---------------------------------------------------------------------------
// With the per-day terms (low_memory = false). p_u(t) also holds ufeat_day and su_day
// of the rating's day. A run of equal dates has one su_day, from yfeat_day (the run's
// training items, then the day's pr items, src/tsvdx4p.rs:500-527), and its error
// sum over sqrt(day count) goes to every item of the run as a yfeat_day delta
// (:614-622).
//
// A user's ratings come in item order as a rule, so nearly every run is one rating
// whose su_day is its item's row and whose delta goes to that item alone. Two such
// ratings make a pair as above (of two days: neither's ufeat_day is the other's);
// every other rating is taken alone. The item rows come through the ring; a
// rating's ufeat_day row is asked for a pair ahead, and taken from the registers of
// the ratings in between where they train the same day.
//
// A user of many ratings is a chain that bounds the pass (7,233 of 6 M), so registers
// go before warps: 5, 4, 3 and 2 blocks an SM at f = 60 took 6.2 (400 bytes spilled),
// 4.5, 4.2 and 4.0 ms, one rating at a time with every row waited for 17.9 ms (one
// B200, CUDA events; 6 M ratings, 8,000 items).
// ---------------------------------------------------------------------------
constexpr int day_ctas(int vpl) { return vpl >= 5 ? 2 : 3; }

constexpr int kDayRows = 3;  // rows of a slot: q_i, q^f_{i,fb}, yfeat_day_i

// A yfeat_day delta row, in fixed point: red.global.add.u64.
template <int VPL>
__device__ __forceinline__ void dyd_add(unsigned long long* row, int lane, const Vec<VPL>& x) {
    float f[VPL];
    x.to(f);
#pragma unroll
    for (int v = 0; v < VPL; ++v)
        atomicAdd(row + Row<VPL>::elem(lane, v), (unsigned long long)__double2ll_rn((double)f[v] * kDydScale));
}

// The run of equal dates that starts at record t (its last rating: run1), where it is
// not one rating without pr items: its su_day and sqrt(day count).
template <int VPL>
__device__ __noinline__ void run_rows(const DeviceState& s, uint64_t t, uint64_t run1, uint32_t ud, uint32_t pc, int lane,
                                      Vec<VPL>& sud, float& norm_day) {
    float none = 0.0f;
    sud.zero();
    sum_rows<VPL, false>(s.yfeat_day, nullptr, nullptr, s.Fs, run1 - t + 1,
                         [&](uint64_t q) { return rec_id(__ldg(&s.rec[t + q].key)); }, lane, sud, none);
    if (pc) {
        const uint32_t* list = s.ud_list_item + s.ud_list_off[ud];
        sum_rows<VPL, false>(s.yfeat_day, nullptr, nullptr, s.Fs, pc, [&](uint64_t q) { return __ldg(list + q); }, lane, sud,
                             none);
    }
    norm_day = sqrtf((float)((uint32_t)(run1 - t + 1) + pc));
    sud.divide(norm_day);
}

template <int VPL>
__global__ void __launch_bounds__(kUThreads, day_ctas(VPL)) k_user_day_pairs(DeviceState s, EpochParams p,
                                                                             const uint32_t* __restrict__ order,
                                                                             uint32_t n_work) {
    using V = Vec<VPL>;
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF;
    float* ring = smem + (threadIdx.x >> 5) * kRingRows * kDayRows * Fs;
    const bool ordinal = s.raw != nullptr;
    // decays as in k_user_pairs
    const float da = -p.lr_u * p.reg_u, db = -p.lr_u2 * p.reg_u2, dc = -p.lr_cu * p.reg_cu, dh = -p.lr_ud * p.reg_ud;
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
        const uint64_t total = (end - start) + (p.full_su ? (s.pr_off[u + 1] - s.pr_off[u]) : 0);
        const float norm = sqrtf((float)total);
        V su;
        float sub;
        load_su<VPL>(s, p, Bf16Copies{}, u, start, end, norm, lane, su, sub);
        V pu, p2, seq;
        pu.load_cg(s.ufeat + (size_t)u * Fs, lane);
        p2.load_cg(s.ufeat2 + (size_t)u * Fs, lane);
        seq.zero();
        float ub = __ldcg(s.ubias + u), al = __ldcg(s.alpha_u + u);
        float cm = __ldcg(s.cu + u) - 1.0f;  // c_u - 1
        float bb0 = lane < (int)T ? __ldcg(s.but_bin + (size_t)u * T + lane) : 0.0f;
        float bb1 = lane + 32 < (int)T ? __ldcg(s.but_bin + (size_t)u * T + 32 + lane) : 0.0f;
        float sum_err = 0.0f;
        // a longer run's su_day and error sum; ufeat_day of the next two ratings
        V sud, seqd, pn0, pn1;
        float norm_day = 1.0f;
        uint64_t run0 = 0, run1 = 0;
        pn0.zero();
        pn1.zero();

        auto chunk_rec = [&](uint64_t base) { return load_rec(s.rec + min(base + lane, end - 1)); };
        Rec ahead = chunk_rec(start);
        // rating j of the chunk whose keys are `keys` into slot j % kRingRows: q_i, q^f_{i,fb}
        auto ask = [&](uint32_t keys, uint32_t j) {
            const uint32_t key = __shfl_sync(kFull, keys, j);
            float* slot = ring + (j % kRingRows) * kDayRows * Fs;
            row_cp_async<VPL>(slot, s.ifeat + (size_t)rec_id(key) * Fs, lane);
            row_cp_async<VPL>(slot + Fs, s.ifeat_freq + ((size_t)rec_id(key) * NF + rec_fbin(key)) * Fs, lane);
            row_cp_async<VPL>(slot + 2 * Fs, s.yfeat_day + (size_t)rec_id(key) * Fs, lane);
            cp_async_commit();
        };
#pragma unroll 1
        for (int q = 0; q < kAheadRows; ++q) ask(ahead.key, q);
        uint32_t last_ud = 0xffffffffu;  // of the rating before the chunk
        if (p.has_ud) {
            pn0.load_cg(s.ufeat_day + (size_t)__shfl_sync(kFull, ahead.ud, 0) * Fs, lane);
            pn1.load_cg(s.ufeat_day + (size_t)__shfl_sync(kFull, ahead.ud, 1) * Fs, lane);
        }
        for (uint64_t base = start; base < end; base += 32) {
            const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
            const Rec r = ahead;
            ahead = chunk_rec(base + 32);
            const uint32_t i = rec_id(r.key), tb = rec_tbin(r.key);
            const float bi = __ldg(s.ibias + i) + __ldg(s.bit_bin + (size_t)i * T + tb) +
                             __ldg(s.ibias_freq + (size_t)i * NF + rec_fbin(r.key));
            const float ct = __ldg(s.cut + r.ud);
            const uint32_t pr_day = p.full_su ? __ldg(s.ud_pr_cnt + r.ud) : 0u;
            // the day's and the time bin's bias, kept current for every rating of the chunk
            float bud = __ldcg(s.ubias_day + r.ud), but;
            {
                const float x0 = __shfl_sync(kFull, bb0, tb & 31), x1 = __shfl_sync(kFull, bb1, tb & 31);
                but = tb < 32 ? x0 : x1;
            }
            const float c0 = s.gbias + sub + bi * (1.0f + ct) - (ordinal ? 0.0f : r.res);
            // M's parts for this lane's rating and the next one's: M = mb + mg qe_0 . qe_1
            float mb, mg;
            unsigned firsts, lasts, lone;  // of their runs; runs of one rating without pr items
            {
                const float dn = __shfl_down_sync(kFull, r.dev, 1), bn = __shfl_down_sync(kFull, bi, 1);
                const uint32_t tn = __shfl_down_sync(kFull, tb, 1);
                const float dd = r.dev * dn;
                mb = p.lr_ub + p.lr_ta * dd + (tn == tb ? p.lr_tu : 0.0f) + p.lr_cu * (bi * bn);
                mg = p.lr_u + p.lr_u2 * dd;
                uint32_t before = __shfl_up_sync(kFull, r.ud, 1), after = __shfl_down_sync(kFull, r.ud, 1);
                const uint32_t next = __shfl_sync(kFull, ahead.ud, 0);
                if (lane == 0) before = last_ud;
                if (lane == 31) after = next;
                firsts = __ballot_sync(kFull, before != r.ud);
                lasts = __ballot_sync(kFull, after != r.ud || base + lane + 1 >= end);
                lone = __ballot_sync(kFull, pr_day == 0) & firsts & lasts;
                last_ud = __shfl_sync(kFull, r.ud, 31);
            }
#pragma unroll 1
            for (uint32_t j = 0; j < cnt;) {
                const bool alone = lone >> j & 1u;
                const bool two = alone && j + 1 < cnt && (lone >> (j + 1) & 1u);
                const uint32_t j1 = two ? j + 1 : j, step = two ? 2 : 1;
                const uint32_t ud0 = __shfl_sync(kFull, r.ud, j), ud1 = __shfl_sync(kFull, r.ud, j1);
                if (!alone && (firsts >> j & 1u)) {
                    const unsigned to = lasts & (0xffffffffu << j);
                    run0 = base + j;
                    run1 = to ? base + __ffs((int)to) - 1 : base + 31;
                    while (!to) {  // past the chunk: 32 records at a time
                        const uint64_t at = run1 + 1 + lane;
                        const unsigned past = __ballot_sync(kFull, at >= end || __ldg(&s.rec[at].ud) != ud0);
                        if (past) {
                            run1 += __ffs((int)past) - 1;
                            break;
                        }
                        run1 += 32;
                    }
                    run_rows<VPL>(s, run0, run1, ud0, __shfl_sync(kFull, pr_day, j), lane, sud, norm_day);
                    seqd.zero();
                }
                cp_async_wait<kAheadRows - 2>();
                V q0, q1, x0, x1;  // the ratings' rows; their su + su_day + ufeat_day
                {
                    const float* slot = ring + (j % kRingRows) * kDayRows * Fs;
                    V f;
                    q0.load(slot, lane);
                    f.load(slot + Fs, lane);
                    q0.add(f);
                    x0 = sud;
                    if (alone) x0.load(slot + 2 * Fs, lane);
                    x0.add(su);
                    x0.add(pn0);
                    slot = ring + (j1 % kRingRows) * kDayRows * Fs;
                    q1.load(slot, lane);
                    f.load(slot + Fs, lane);
                    q1.add(f);
                    x1.load(slot + 2 * Fs, lane);
                    x1.add(su);
                    x1.add(pn1);
                }
                V p0 = pn0, p1 = pn1;
                // ufeat_day of the next two ratings (the last's again past the end)
                const uint32_t n0 = j + step, n1 = n0 + 1;
                const uint32_t nd0 = __shfl_sync(kFull, n0 < 32 ? r.ud : ahead.ud, n0 & 31);
                const uint32_t nd1 = __shfl_sync(kFull, n1 < 32 ? r.ud : ahead.ud, n1 & 31);
                if (p.has_ud) {
                    pn0.load_cg(s.ufeat_day + (size_t)nd0 * Fs, lane);
                    pn1.load_cg(s.ufeat_day + (size_t)nd1 * Fs, lane);
                }
                // as many rows more, of the next chunk where this one ends
#pragma unroll 1
                for (uint32_t q = j + kAheadRows; q < j + kAheadRows + step; ++q)
                    ask(q < 32 ? r.key : ahead.key, q & 31u);
                const float d0 = __shfl_sync(kFull, r.dev, j), d1 = __shfl_sync(kFull, r.dev, j1);
                float v0, v1, g = q0.dot(q1);
                {
                    x0.fma(d0, p2);
                    x0.add(pu);
                    v0 = q0.dot(x0);
                    x1.fma(b1 * d1, p2);
                    x1.fma(a1, pu);
                    v1 = q1.dot(x1);
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
                const float bi0 = __shfl_sync(kFull, bi, j), bi1 = __shfl_sync(kFull, bi, j1);
                float e0 = __shfl_sync(kFull, cl, j) + ub + al * d0 + bi0 * cm + v0;
                float e1 = __shfl_sync(kFull, cl, j1) + ub + al * d1 + bi1 * (c1 * cm) + v1;
                const float m10 = __shfl_sync(kFull, mb, j) + __shfl_sync(kFull, mg, j) * g;
                if (ordinal) e0 = ordinal_err(s.thresholds, e0, (int)__shfl_sync(kFull, r.res, j));
                e1 = fmaf(-m10, e0, e1);
                if (ordinal) e1 = ordinal_err(s.thresholds, e1, (int)__shfl_sync(kFull, r.res, j1));
                // a rating taken alone: no update and no decay from the second
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
                if (p.has_ud) {
                    t = p0;
                    t.scale(dh);
                    t.fma(-p.lr_ud * e0, q0);
                    p0.add(t);
                    p0.store_cg(s.ufeat_day + (size_t)ud0 * Fs, lane);
                    if (two) {
                        t = p1;
                        t.scale(dh);
                        t.fma(-p.lr_ud * e1, q1);
                        p1.add(t);
                        p1.store_cg(s.ufeat_day + (size_t)ud1 * Fs, lane);
                    }
                    // (asked for before these)
                    if (nd0 == ud0) pn0 = p0;
                    if (nd1 == ud0) pn1 = p0;
                    if (two && nd0 == ud1) pn0 = p1;
                    if (two && nd1 == ud1) pn1 = p1;
                }
                sum_err += e0;
                sum_err += e1;
                ub -= p.lr_ub * (e0 + e1);
                al -= p.lr_ta * fmaf(e0, d0, e1 * d1);
                cm = fmaf(two ? dc2 : dc, cm, cm) - p.lr_cu * fmaf(c2 * e0, bi0, e1 * bi1);
                bud -= p.lr_ubd * ((ud0 == r.ud ? e0 : 0.0f) + (two && ud1 == r.ud ? e1 : 0.0f));
                if (p.lr_tu != 0.0f) {
                    const uint32_t t0 = __shfl_sync(kFull, tb, j), t1 = __shfl_sync(kFull, tb, j1);
                    but -= p.lr_tu * ((t0 == tb ? e0 : 0.0f) + (t1 == tb ? e1 : 0.0f));
                    const uint32_t lo = lane, hi = lane + 32;
                    bb0 -= p.lr_tu * ((t0 == lo ? e0 : 0.0f) + (t1 == lo ? e1 : 0.0f));
                    bb1 -= p.lr_tu * ((t0 == hi ? e0 : 0.0f) + (t1 == hi ? e1 : 0.0f));
                }
                // yfeat_day deltas: a lone rating's to its item, a longer run's at its end
                if (alone) {
                    const uint32_t i0 = __shfl_sync(kFull, i, j), i1 = __shfl_sync(kFull, i, j1);
                    q0.scale(e0);
                    dyd_add<VPL>(s.dyd_fix + (size_t)i0 * Fs, lane, q0);
                    if (two) {
                        q1.scale(e1);
                        dyd_add<VPL>(s.dyd_fix + (size_t)i1 * Fs, lane, q1);
                    }
                } else {
                    seqd.fma(e0, q0);
                    if (base + j == run1) {
                        seqd.divide(norm_day);
#pragma unroll 1
                        for (uint64_t q = run0; q <= run1; ++q)
                            dyd_add<VPL>(s.dyd_fix + (size_t)rec_id(__ldg(&s.rec[q].key)) * Fs, lane, seqd);
                    }
                }
                j += step;
            }
            // the chunk's day biases (ratings of one day hold the same value)
            __stcg(s.ubias_day + r.ud, bud);
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

template <int VPL>
void launch_days(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n) {
    auto kern = k_user_day_pairs<VPL>;
    const size_t smem = (size_t)(kUThreads / 32) * kRingRows * kDayRows * s.Fs * sizeof(float);
    int dev = 0, sms = 0, per_sm = 0;
    allow_dyn_smem(kern, smem);
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
