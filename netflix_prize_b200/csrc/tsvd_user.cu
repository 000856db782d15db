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

}  // namespace tsvd
