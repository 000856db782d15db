// The strata for rows of more than 256 columns (low_memory, FP32, no
// ordinal head): the chains of
// tsvd_user.cu and tsvd_item.cuh, ratings two at a time, with a block per user or
// item. Warp w of the block holds columns 128 w .. 128 w + 127 of the unit's rows in
// registers; a pair's three sums meet in shared memory behind one barrier, and every
// warp then has the pair's errors. The scalars (records, biases) are kept by every
// warp alike, so nothing else is exchanged.
//
// A unit's chain bounds the pass (9,959 ratings of the most rated of 3,001 items): one
// warp that reads and writes its rows in memory, slice by slice, twice a rating
// takes 1.7 us a rating at 512 columns, a block 0.3. 2 M ratings, f = 400: user pass
// 6.0 -> 1.1 ms, item pass 16.7 -> 2.9 ms (one B200, CUDA events). Two warps of 256
// columns for four of 128 took 1.3 and 4.0 (the latter against 3.5).
//
// Blocks of up to 16 warps keep the registers of these chains: rows up to 2,048
// columns. Wider ones take a warp per unit (tsvd_strat.cu).
#include "tsvd_item.cuh"

namespace tsvd {
namespace {

constexpr int kWideV = 4;                       // a lane's values
constexpr uint32_t kWarpCols = 32 * kWideV;     // a warp's columns
constexpr int kWideWarps = 16;                  // most warps of a block
constexpr uint32_t kWideRows = 8, kWideAhead = 6;  // the user pass: ratings in the ring, asked for ahead
constexpr size_t kWideSmem = 224 * 1024;        // of the 227 KB a block can have
constexpr uint32_t kSumFloats = 2 * 3 * kWideWarps;

using W4 = Vec<kWideV>;

// The block's sums of three values per lane, `sums` one of two buffers in turn (a
// buffer's last readers are past the barrier of the other one).
__device__ __forceinline__ void block_sums(float* sums, int lane, int warp, int warps, float& a, float& b, float& g) {
    {
        const bool up = (lane & 16) != 0;
        const float keep = up ? b : a, send = up ? a : b;
        a = keep + __shfl_xor_sync(kFull, send, 16);
        g += __shfl_xor_sync(kFull, g, 16);
        const bool up8 = (lane & 8) != 0;
        const float keep8 = up8 ? g : a, send8 = up8 ? a : g;
        a = keep8 + __shfl_xor_sync(kFull, send8, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    }
    // lanes 0, 16 and 8 hold a, b and g
    if ((lane & 7) == 0 && lane < 24) sums[(lane == 0 ? 0 : lane == 16 ? 1 : 2) * kWideWarps + warp] = a;
    __syncthreads();
    a = b = g = 0.0f;
    for (int w = 0; w < warps; w += 2) {  // (an even number of warps)
        const float2 x = *reinterpret_cast<const float2*>(sums + w);
        const float2 y = *reinterpret_cast<const float2*>(sums + kWideWarps + w);
        const float2 z = *reinterpret_cast<const float2*>(sums + 2 * kWideWarps + w);
        a += x.x + x.y;
        b += y.x + y.y;
        g += z.x + z.y;
    }
}

__global__ void __launch_bounds__(32 * kWideWarps) k_user_wide_pairs(DeviceState s, EpochParams p,
                                                                     const uint32_t* __restrict__ order, uint32_t n_work) {
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float sums[kSumFloats];
    __shared__ uint32_t sh_k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF, col0 = warp * kWarpCols;
    float* ring = smem + col0;
    // decays as in k_user_pairs
    const float da = -p.lr_u * p.reg_u, db = -p.lr_u2 * p.reg_u2, dc = -p.lr_cu * p.reg_cu;
    const float a1 = 1.0f + da, b1 = 1.0f + db, c1 = 1.0f + dc;
    const float da2 = fmaf(da, da, 2.0f * da), db2 = fmaf(db, db, 2.0f * db), dc2 = fmaf(dc, dc, 2.0f * dc);
    uint32_t turn = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sh_k = atomicAdd(&s.counters[0], 1u);
        __syncthreads();
        const uint32_t k = sh_k;
        if (k >= n_work) break;
        const uint32_t u = order[k];
        const uint64_t start = s.user_off[u], end = s.user_off[u + 1];
        if (start == end) continue;
        const uint64_t ps = s.pr_off[u], pe = s.pr_off[u + 1];
        const float norm = sqrtf((float)((end - start) + (p.full_su ? (pe - ps) : 0)));
        // su (src/tsvdx4p.rs:466-491): equals ycache[u] bit for bit when full_su
        // holds and ycache was rebuilt from the current y.
        W4 su;
        float sub;
        if (p.use_ycache) {
            su.load_cg(s.ycache + (size_t)u * Fs + col0, lane);
            sub = __ldcg(s.ycache_bias + u);
        } else {
            su.zero();
            sub = 0.0f;
            const Rec* rr = s.rec + start;
            const uint32_t* pp = s.pr_item + ps;
            sum_rows<kWideV, false>(s.yfeat + col0, nullptr, s.ybias, Fs, end - start,
                                    [&](uint64_t q) { return rec_id(__ldg(&rr[q].key)); }, lane, su, sub);
            sum_rows<kWideV, false>(s.yfeat + col0, nullptr, s.ybias, Fs, p.full_su ? pe - ps : 0,
                                    [&](uint64_t q) { return __ldg(pp + q); }, lane, su, sub);
            su.divide(norm);
            sub = sub / norm;
            su.store_cg(s.ycache + (size_t)u * Fs + col0, lane);
            if (threadIdx.x == 0) s.ycache_bias[u] = sub;
        }
        W4 pu, p2, seq;
        pu.load_cg(s.ufeat + (size_t)u * Fs + col0, lane);
        p2.load_cg(s.ufeat2 + (size_t)u * Fs + col0, lane);
        seq.zero();
        float ub = __ldcg(s.ubias + u), al = __ldcg(s.alpha_u + u);
        float cm = __ldcg(s.cu + u) - 1.0f;  // c_u - 1
        float bb0 = lane < (int)T ? __ldcg(s.but_bin + (size_t)u * T + lane) : 0.0f;
        float bb1 = lane + 32 < (int)T ? __ldcg(s.but_bin + (size_t)u * T + 32 + lane) : 0.0f;
        float sum_err = 0.0f;
        auto chunk_rec = [&](uint64_t base) { return load_rec(s.rec + min(base + lane, end - 1)); };
        Rec ahead = chunk_rec(start);
        auto ask = [&](uint32_t keys, uint32_t j) {
            const uint32_t i = rec_id(__shfl_sync(kFull, keys, j));
            row_cp_async<kWideV>(ring + (j % kWideRows) * Fs, s.qe0 + (size_t)i * Fs + col0, lane);
        };
#pragma unroll
        for (uint32_t q = 0; q < kWideAhead; q += 2) {
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
                const float x0 = __shfl_sync(kFull, bb0, tb & 31), x1 = __shfl_sync(kFull, bb1, tb & 31);
                but = tb < 32 ? x0 : x1;
            }
            const float c0 = s.gbias + sub + bi * (1.0f + ct) - r.res;
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
                    const bool here = j + kWideAhead < 32;
                    const uint32_t keys = here ? r.key : ahead.key, q = (j + kWideAhead) & 31u;
                    ask(keys, q);
                    ask(keys, q + 1);
                    cp_async_commit();
                }
                cp_async_wait<kWideAhead / 2>();
                W4 q0, q1;
                q0.load(ring + (j % kWideRows) * Fs, lane);
                q1.load(ring + ((j + 1) % kWideRows) * Fs, lane);
                const bool two = j + 1 < cnt;
                const float d0 = __shfl_sync(kFull, r.dev, j), d1 = __shfl_sync(kFull, r.dev, j + 1);
                float v0, v1, g = q0.dot(q1);
                {
                    W4 t = su;
                    t.fma(d0, p2);
                    t.add(pu);
                    v0 = q0.dot(t);
                    t = su;
                    t.fma(b1 * d1, p2);
                    t.fma(a1, pu);
                    v1 = q1.dot(t);
                }
                block_sums(sums + (turn++ & 1) * 3 * kWideWarps, lane, warp, warps, v0, v1, g);
                const float cl = c0 + but + bud;
                const float bi0 = __shfl_sync(kFull, bi, j), bi1 = __shfl_sync(kFull, bi, j + 1);
                float e0 = __shfl_sync(kFull, cl, j) + ub + al * d0 + bi0 * cm + v0;
                float e1 = __shfl_sync(kFull, cl, j + 1) + ub + al * d1 + bi1 * (c1 * cm) + v1;
                const float m10 = __shfl_sync(kFull, mb, j) + __shfl_sync(kFull, mg, j) * g;
                e1 = fmaf(-m10, e0, e1);
                // a last rating without a second: no update and no decay from it
                e1 = two ? e1 : 0.0f;
                const float a2 = two ? a1 : 1.0f, b2 = two ? b1 : 1.0f, c2 = two ? c1 : 1.0f;
                seq.fma(e0, q0);
                seq.fma(e1, q1);
                W4 t = pu;
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
            // the chunk's day biases (ratings of one day hold the same value). A day
            // may come back in the next chunk: no warp reads it there before warp 0 has
            // written it, nor has one yet to read this chunk's when warp 0 writes
            // (they have all passed the chunk's first barrier).
            if (warp == 0 && hud) __stcg(s.ubias_day + r.ud, bud);
            __syncthreads();
        }
        cp_async_wait<0>();
        pu.store_cg(s.ufeat + (size_t)u * Fs + col0, lane);
        p2.store_cg(s.ufeat2 + (size_t)u * Fs + col0, lane);
        seq.divide(norm);
        seq.store_cg(s.g_user + (size_t)u * Fs + col0, lane);
        if (warp == 0) {
            if (lane == 0) {
                s.ubias[u] = ub;
                s.alpha_u[u] = al;
                s.cu[u] = cm + 1.0f;
                s.e_user[u] = sum_err / norm;
            }
            if (lane < (int)T) s.but_bin[(size_t)u * T + lane] = bb0;
            if (lane + 32 < (int)T) s.but_bin[(size_t)u * T + 32 + lane] = bb1;
        }
    }
}

// QS: the item's q^f rows are kept in shared memory; in the table they come back
// through L2 within the chain. ROWS: ratings in the ring, asked for ROWS - 2 ahead.
// (2 M ratings, 512 columns: 4.6 ms with 8 rows and the table, 3.5 with the q^f rows
// in shared memory, 2.9 with 16 rows as well.)
template <bool QS, uint32_t ROWS>
__global__ void __launch_bounds__(32 * kWideWarps) k_item_wide_pairs(DeviceState s, EpochParams p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float sums[kSumFloats];
    __shared__ uint32_t sh_k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF, col0 = warp * kWarpCols;
    float* ring = smem + col0;
    const float da = row_decay(p.lr_i, p.reg_i, false), df = row_decay(p.lr_iqf, p.reg_iqf, false);
    const float a1 = 1.0f + da, f1 = 1.0f + df;
    const float da2 = fmaf(da, da, 2.0f * da), df2 = fmaf(df, df, 2.0f * df);
    uint32_t turn = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sh_k = atomicAdd(&s.counters[2], 1u);
        __syncthreads();
        const uint32_t k = sh_k;
        if (k >= s.n_item_work) break;
        const uint32_t i = s.item_work[k];
        const uint64_t start = s.item_off[i], end = s.item_off[i + 1];
        if (start == end) continue;
        W4 q;
        q.load_cg(s.ifeat + (size_t)i * Fs + col0, lane);
        // (each lane reads back only what it wrote)
        float* qf_row = s.ifeat_freq + (size_t)i * NF * Fs + col0;
        float* qf = QS ? smem + (size_t)ROWS * 2 * Fs + col0 : qf_row;
        if constexpr (QS)
            for (uint32_t b = 0; b < NF; ++b) row_cp_async<kWideV>(qf + b * Fs, qf_row + (size_t)b * Fs, lane);
        float ib = __ldcg(s.ibias + i);
        float bt0 = lane < (int)T ? __ldcg(s.bit_bin + (size_t)i * T + lane) : 0.0f;
        float bt1 = lane + 32 < (int)T ? __ldcg(s.bit_bin + (size_t)i * T + 32 + lane) : 0.0f;
        float bf0 = lane < (int)NF ? __ldcg(s.ibias_freq + (size_t)i * NF + lane) : 0.0f;
        float bf1 = lane + 32 < (int)NF ? __ldcg(s.ibias_freq + (size_t)i * NF + 32 + lane) : 0.0f;
        auto chunk_rec = [&](uint64_t base) { return load_rec(s.irec + min(base + lane, end - 1)); };
        Rec ahead = chunk_rec(start);
        auto ask = [&](uint32_t keys, uint32_t j) {
            const uint32_t u = rec_id(__shfl_sync(kFull, keys, j));
            float* slot = ring + (j % ROWS) * 2 * Fs;
            row_cp_async<kWideV>(slot, s.pyc + (size_t)u * Fs + col0, lane);
            row_cp_async<kWideV>(slot + Fs, s.ufeat2 + (size_t)u * Fs + col0, lane);
        };
#pragma unroll
        for (uint32_t e = 0; e < (ROWS - 2); e += 2) {
            ask(ahead.key, e);
            ask(ahead.key, e + 1);
            cp_async_commit();
        }
        for (uint64_t base = start; base < end; base += 32) {
            const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
            const Rec r = ahead;
            ahead = chunk_rec(base + 32);
            const uint32_t tb = rec_tbin(r.key), fb = rec_fbin(r.key);
            float cu, c0;
            {
                float bu;
                user_scalars(s, r, bu, cu);
                c0 = s.gbias + bu - r.res;
            }
            // M's parts for this lane's rating and the next one's: M = mb + mg pe_0 . pe_1
            float mb, mg;
            {
                const float cn = __shfl_down_sync(kFull, cu, 1);
                const uint32_t tn = __shfl_down_sync(kFull, tb, 1), fn = __shfl_down_sync(kFull, fb, 1);
                mb = cu * cn * (p.lr_ib + (tn == tb ? p.lr_ti : 0.0f) + (fn == fb ? p.lr_ibf : 0.0f));
                mg = p.lr_i + (fn == fb ? p.lr_iqf : 0.0f);
            }
#pragma unroll 1
            for (uint32_t j = 0; j < cnt; j += 2) {
                {  // two ratings' rows more, of the next chunk where this one ends
                    const bool here = j + (ROWS - 2) < 32;
                    const uint32_t keys = here ? r.key : ahead.key, e = (j + (ROWS - 2)) & 31u;
                    ask(keys, e);
                    ask(keys, e + 1);
                    cp_async_commit();
                }
                const uint32_t fb0 = __shfl_sync(kFull, fb, j), fb1 = __shfl_sync(kFull, fb, j + 1);
                const bool two = j + 1 < cnt, same = fb0 == fb1 && two;
                float* r0 = qf + (size_t)fb0 * Fs;
                float* r1 = qf + (size_t)fb1 * Fs;
                W4 g0, g1;
                if constexpr (!QS) {
                    g0.load(r0, lane);
                    g1.load(r1, lane);
                }
                cp_async_wait<(ROWS - 2) / 2>();
                if constexpr (QS) {
                    g0.load(r0, lane);
                    g1.load(r1, lane);
                }
                auto pe = [&](uint32_t e, W4& x) {  // p_u + ycache_u + dev p2_u of rating e
                    W4 y;
                    const float* slot = ring + (e % ROWS) * 2 * Fs;
                    x.load(slot, lane);
                    y.load(slot + Fs, lane);
                    x.fma(__shfl_sync(kFull, r.dev, e), y);
                };
                W4 x0, x1;
                pe(j, x0);
                pe(j + 1, x1);
                float g = x0.dot(x1), v0, v1;
                {
                    W4 t = g0;
                    t.add(q);
                    v0 = x0.dot(t);
                    t = g1;
                    if (same) t.scale(f1);
                    t.fma(a1, q);
                    v1 = x1.dot(t);
                }
                block_sums(sums + (turn++ & 1) * 3 * kWideWarps, lane, warp, warps, v0, v1, g);
                const uint32_t tb0 = __shfl_sync(kFull, tb, j), tb1 = __shfl_sync(kFull, tb, j + 1);
                const float cu0 = __shfl_sync(kFull, cu, j), cu1 = __shfl_sync(kFull, cu, j + 1);
                const float bi0 = ib + __shfl_sync(kFull, tb0 < 32 ? bt0 : bt1, tb0 & 31) +
                                  __shfl_sync(kFull, fb0 < 32 ? bf0 : bf1, fb0 & 31);
                const float bi1 = ib + __shfl_sync(kFull, tb1 < 32 ? bt0 : bt1, tb1 & 31) +
                                  __shfl_sync(kFull, fb1 < 32 ? bf0 : bf1, fb1 & 31);
                float e0 = __shfl_sync(kFull, c0, j) + bi0 * cu0 + v0;
                float e1 = __shfl_sync(kFull, c0, j + 1) + bi1 * cu1 + v1;
                const float m10 = __shfl_sync(kFull, mb, j) + __shfl_sync(kFull, mg, j) * g;
                e1 = fmaf(-m10, e0, e1);
                // a last rating without a second: no update and no decay from it
                e1 = two ? e1 : 0.0f;
                const float a2 = two ? a1 : 1.0f;
                // each row's change is summed first and rounded into the row once
                {
                    W4 t = q;
                    t.scale(two ? da2 : da);
                    t.fma(-p.lr_i * a2 * e0, x0);
                    t.fma(-p.lr_i * e1, x1);
                    q.add(t);
                }
                {
                    W4 t = g0;
                    t.scale(same ? df2 : df);
                    t.fma(-p.lr_iqf * (same ? f1 : 1.0f) * e0, x0);
                    if (same) t.fma(-p.lr_iqf * e1, x1);
                    g0.add(t);
                    g0.store(r0, lane);
                }
                if (two && !same) {
                    W4 t = g1;
                    t.scale(df);
                    t.fma(-p.lr_iqf * e1, x1);
                    g1.add(t);
                    g1.store(r1, lane);
                }
                const float w0 = e0 * cu0, w1 = e1 * cu1;
                ib -= p.lr_ib * (w0 + w1);
                const uint32_t lo = lane, hi = lane + 32;
                bt0 -= p.lr_ti * ((tb0 == lo ? w0 : 0.0f) + (tb1 == lo ? w1 : 0.0f));
                bf0 -= p.lr_ibf * ((fb0 == lo ? w0 : 0.0f) + (fb1 == lo ? w1 : 0.0f));
                if (T > 32) bt1 -= p.lr_ti * ((tb0 == hi ? w0 : 0.0f) + (tb1 == hi ? w1 : 0.0f));
                if (NF > 32) bf1 -= p.lr_ibf * ((fb0 == hi ? w0 : 0.0f) + (fb1 == hi ? w1 : 0.0f));
            }
        }
        cp_async_wait<0>();
        q.store_cg(s.ifeat + (size_t)i * Fs + col0, lane);
        if constexpr (QS)
            for (uint32_t b = 0; b < NF; ++b) {
                W4 x;
                x.load(qf + b * Fs, lane);
                x.store_cg(qf_row + (size_t)b * Fs, lane);
            }
        if (warp == 0) {
            if (lane == 0) s.ibias[i] = ib;
            if (lane < (int)T) s.bit_bin[(size_t)i * T + lane] = bt0;
            if (lane + 32 < (int)T) s.bit_bin[(size_t)i * T + 32 + lane] = bt1;
            if (lane < (int)NF) s.ibias_freq[(size_t)i * NF + lane] = bf0;
            if (lane + 32 < (int)NF) s.ibias_freq[(size_t)i * NF + 32 + lane] = bf1;
        }
    }
}

template <class Kern>
unsigned wide_grid(Kern kern, uint32_t Fs, size_t smem) {
    int dev = 0, sms = 0, per_sm = 0;
    allow_dyn_smem(kern, smem);
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TSVD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)(Fs / kWideV), smem));
    return (unsigned)(sms * std::max(per_sm, 1));
}

}  // namespace

bool wide_pairs_fit(uint32_t Fs) { return Fs > 256 && Fs <= kWideWarps * kWarpCols; }

void launch_user_wide_pairs(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n) {
    const size_t smem = (size_t)kWideRows * s.Fs * sizeof(float);
    const unsigned g = wide_grid(k_user_wide_pairs, s.Fs, smem);
    k_user_wide_pairs<<<g, s.Fs / kWideV, smem, m->stream>>>(s, p, work, n);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

void launch_item_wide_pairs(tsvd_model* m, const DeviceState& s, const EpochParams& p) {
    // what fits of the q^f rows and a ring of 16 ratings, the rows first
    const size_t slot = 2 * s.Fs * sizeof(float), rows = (size_t)s.NF * s.Fs * sizeof(float);
    const bool qs = 8 * slot + rows <= kWideSmem, deep = qs && 16 * slot + rows <= kWideSmem;
    const size_t smem = (deep ? 16 : 8) * slot + (qs ? rows : 0);
    auto kern = deep ? k_item_wide_pairs<true, 16> : qs ? k_item_wide_pairs<true, 8> : k_item_wide_pairs<false, 8>;
    const unsigned g = wide_grid(kern, s.Fs, smem);
    kern<<<g, s.Fs / kWideV, smem, m->stream>>>(s, p);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

}  // namespace tsvd
