// The item stratum's light items (tsvd_item.cu, tsvd_item_tiles.cu).
#pragma once
#include <cuda_fp16.h>

#include "tsvd_chain.cuh"

namespace tsvd {

// a - 1 for a row's decay factor a = 1 - lr reg, or for that factor rounded to FP32
// (once: the product is not rounded before it).
__device__ __forceinline__ float row_decay(float lr, float reg, bool rounded) {
    return rounded ? __fmaf_rn(-lr, reg, 1.0f) - 1.0f : -(lr * reg);
}

// Four tables of 36 floats: a_i^n, a_f^n, a_i^n - 1, a_f^n - 1 for n = 0 .. N. The
// rounded factors' powers are products in FP32, as those items have had them.
template <int N>
__device__ __forceinline__ void decay_powers(float* pow, const EpochParams& p, bool rounded) {
    const float d_i = row_decay(p.lr_i, p.reg_i, rounded), d_f = row_decay(p.lr_iqf, p.reg_iqf, rounded);
    float x = 0.0f, y = 0.0f;  // a^n - 1 = (a^(n-1) - 1) a + (a - 1)
    for (int e = 0; e <= N; ++e) {
        pow[e] = 1.0f + x;
        pow[36 + e] = 1.0f + y;
        pow[72 + e] = x;
        pow[108 + e] = y;
        x = rounded ? __fmul_rn(1.0f + x, 1.0f + d_i) - 1.0f : fmaf(x, d_i, x) + d_i;
        y = rounded ? __fmul_rn(1.0f + y, 1.0f + d_f) - 1.0f : fmaf(y, d_f, y) + d_f;
    }
}

// The per-rating a - 1 whose 32nd power is that table's: what a chain of single
// ratings applies to an item with the rounded factors.
__device__ __forceinline__ float rounded_step(float d) {
    float x = 1.0f;
    for (int e = 0; e < 32; ++e) x = __fmul_rn(x, 1.0f + d);
    double r = x;
    for (int e = 0; e < 5; ++e) r = sqrt(r);
    return (float)(r - 1.0);
}

// ---------------------------------------------------------------------------
// The dots pe_i . pe_k of a round by the warp-level MMAs, with the digits of FP32
// products: a value is taken as the sum of two FP16 parts, 22 bits, and of the four
// products all but the least. A row is scaled by a power of two first, its largest
// value to 2^14 .. 2^15, so that a part's 2^-25 is at most 2^-39 of that value. (Two
// BF16 parts hold 16 bits: the next rating's error was up to 2^-15 lr |pe_i||pe_k| of the
// last one off. 25 M ratings, f = 256: item pass 15.0 ms with those, 15.7 with these;
// three BF16 parts and six products 9 % more. Up to 128 columns within 6 % either way: 1
// M, f = 32, 0.60 and 0.59 ms; per-day 6 M, 4.13 and 4.02; 1 M, f = 128, 0.86 and 0.91.)
// ---------------------------------------------------------------------------
// A warp's row: the inverse of its scale. (Rows below 2^-112 are scaled as that.)
template <int VPL>
__device__ __forceinline__ float row_unscale(const float (&x)[VPL]) {
    float m = fabsf(x[0]);
#pragma unroll
    for (int v = 1; v < VPL; ++v) m = fmaxf(m, fabsf(x[v]));
    const uint32_t largest = __reduce_max_sync(kFull, __float_as_uint(m));
    return __uint_as_float((max(largest >> 23, 15u) - 14u) << 23);
}
__device__ __forceinline__ float row_scale(float unscale) { return __uint_as_float(0x7f000000u - __float_as_uint(unscale)); }

// Packed FP16 pairs of (x, y): the values rounded, and what that leaves rounded.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// d (16x8, FP32) += a (16x16, FP16, row-major) . b (16x8, FP16, column-major)
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// An item's biases, spread over a warp.
struct ItemState {
    float ib, bt0, bt1, bf0, bf1;
};

__device__ __forceinline__ ItemState load_item_state(const DeviceState& s, uint32_t i, int lane) {
    const uint32_t T = s.T, NF = s.NF;
    ItemState st;
    st.ib = s.ibias[i];
    st.bt0 = lane < (int)T ? s.bit_bin[(size_t)i * T + lane] : 0.0f;
    st.bt1 = lane + 32 < (int)T ? s.bit_bin[(size_t)i * T + 32 + lane] : 0.0f;
    st.bf0 = lane < (int)NF ? s.ibias_freq[(size_t)i * NF + lane] : 0.0f;
    st.bf1 = lane + 32 < (int)NF ? s.ibias_freq[(size_t)i * NF + 32 + lane] : 0.0f;
    return st;
}

__device__ __forceinline__ void store_item_state(const DeviceState& s, uint32_t i, int lane, const ItemState& st) {
    const uint32_t T = s.T, NF = s.NF;
    if (lane == 0) s.ibias[i] = st.ib;
    if (lane < (int)T) s.bit_bin[(size_t)i * T + lane] = st.bt0;
    if (lane + 32 < (int)T) s.bit_bin[(size_t)i * T + 32 + lane] = st.bt1;
    if (lane < (int)NF) s.ibias_freq[(size_t)i * NF + lane] = st.bf0;
    if (lane + 32 < (int)NF) s.ibias_freq[(size_t)i * NF + 32 + lane] = st.bf1;
}

// ---------------------------------------------------------------------------
// A light item by one warp, its ratings two at a time (as tsvd_user.cu): one
// reduction of three sums, two dots with the item's rows and pe_0 . pe_1. The user
// rows come through a ring of shared-memory slots, q is in registers, the q^f rows
// in the global table (they are the warp's own and stay in L1).
// ---------------------------------------------------------------------------
constexpr int kLightRows = 4;   // ratings in the ring
constexpr int kLightAhead = 2;  // ratings asked for ahead

template <int VPL, bool BF>
__device__ __forceinline__ void item_pairs(const DeviceState& s, const EpochParams& p, const Bf16Copies& bf, uint32_t i,
                                           int lane, float* ring) {
    using V = Vec<VPL>;
    const uint32_t Fs = s.Fs, NF = s.NF, T = s.T;
    const uint64_t start = s.item_off[i], end = s.item_off[i + 1];
    const bool ordinal = s.raw != nullptr;
    const bool rounded = end - start >= s.rounded_decay_min;
    const float di = row_decay(p.lr_i, p.reg_i, rounded), da = rounded ? rounded_step(di) : di, df = row_decay(p.lr_iqf, p.reg_iqf, rounded);
    const float a1 = 1.0f + da, f1 = 1.0f + df;
    const float da2 = fmaf(da, da, 2.0f * da), df2 = fmaf(df, df, 2.0f * df);
    V q;
    q.load_cg(s.ifeat + (size_t)i * Fs, lane);
    float* qf = s.ifeat_freq + (size_t)i * NF * Fs;
    float ib = s.ibias[i];
    float bt0 = lane < (int)T ? s.bit_bin[(size_t)i * T + lane] : 0.0f;
    float bt1 = lane + 32 < (int)T ? s.bit_bin[(size_t)i * T + 32 + lane] : 0.0f;
    float bf0 = lane < (int)NF ? s.ibias_freq[(size_t)i * NF + lane] : 0.0f;
    float bf1 = lane + 32 < (int)NF ? s.ibias_freq[(size_t)i * NF + 32 + lane] : 0.0f;
    auto chunk_rec = [&](uint64_t base) { return load_rec(s.irec + min(base + lane, end - 1)); };
    Rec ahead = chunk_rec(start);
    // a rating's user rows into its slot (BF16 rows are read when they are used)
    auto ask = [&](uint32_t keys, uint32_t j) {
        if constexpr (BF) return;
        const uint32_t u = rec_id(__shfl_sync(kFull, keys, j));
        float* slot = ring + (j % kLightRows) * 2 * Fs;
        row_cp_async<VPL>(slot, s.pyc + (size_t)u * Fs, lane);
        row_cp_async<VPL>(slot + Fs, s.ufeat2 + (size_t)u * Fs, lane);
    };
#pragma unroll
    for (int k = 0; k < kLightAhead; ++k) ask(ahead.key, k);
    cp_async_commit();
    for (uint64_t base = start; base < end; base += 32) {
        const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
        const Rec r = ahead;
        ahead = chunk_rec(base + 32);
        const uint32_t tb = rec_tbin(r.key), fb = rec_fbin(r.key);
        float cu, c0;
        {
            float bu;
            user_scalars(s, r, bu, cu);
            c0 = ordinal ? s.gbias + bu : s.gbias + bu - r.res;
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
                const bool here = j + kLightAhead < 32;
                const uint32_t keys = here ? r.key : ahead.key, k = (j + kLightAhead) & 31u;
                ask(keys, k);
                ask(keys, k + 1);
                cp_async_commit();
            }
            const uint32_t fb0 = __shfl_sync(kFull, fb, j), fb1 = __shfl_sync(kFull, fb, j + 1);
            const bool two = j + 1 < cnt, same = fb0 == fb1 && two;
            float* r0 = qf + (size_t)fb0 * Fs;
            float* r1 = qf + (size_t)fb1 * Fs;
            V g0, g1;
            g0.load(r0, lane);
            g1.load(r1, lane);
            cp_async_wait<1>();
            auto pe = [&](uint32_t k, V& x) {  // p_u + ycache_u + dev p2_u of rating k
                V y;
                if constexpr (BF) {
                    const size_t at = (size_t)rec_id(__shfl_sync(kFull, r.key, k)) * Fs;
                    x.load_bf16(bf.pyc + at, lane);
                    y.load_bf16(bf.ufeat2 + at, lane);
                } else {
                    const float* slot = ring + (k % kLightRows) * 2 * Fs;
                    x.load(slot, lane);
                    y.load(slot + Fs, lane);
                }
                x.fma(__shfl_sync(kFull, r.dev, k), y);
            };
            V x0, x1;
            pe(j, x0);
            pe(j + 1, x1);
            float g = x0.dot(x1), v0, v1;
            {
                V t = g0;
                t.add(q);
                v0 = x0.dot(t);
                t = g1;
                if (same) t.scale(f1);
                t.fma(a1, q);
                v1 = x1.dot(t);
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
            const uint32_t tb0 = __shfl_sync(kFull, tb, j), tb1 = __shfl_sync(kFull, tb, j + 1);
            const float cu0 = __shfl_sync(kFull, cu, j), cu1 = __shfl_sync(kFull, cu, j + 1);
            const float bi0 = ib + __shfl_sync(kFull, tb0 < 32 ? bt0 : bt1, tb0 & 31) +
                              __shfl_sync(kFull, fb0 < 32 ? bf0 : bf1, fb0 & 31);
            const float bi1 = ib + __shfl_sync(kFull, tb1 < 32 ? bt0 : bt1, tb1 & 31) +
                              __shfl_sync(kFull, fb1 < 32 ? bf0 : bf1, fb1 & 31);
            float e0 = __shfl_sync(kFull, c0, j) + bi0 * cu0 + v0;
            float e1 = __shfl_sync(kFull, c0, j + 1) + bi1 * cu1 + v1;
            const float m10 = __shfl_sync(kFull, mb, j) + __shfl_sync(kFull, mg, j) * g;
            if (ordinal) e0 = ordinal_err(s.thresholds, e0, (int)__shfl_sync(kFull, r.res, j));
            e1 = fmaf(-m10, e0, e1);
            if (ordinal) e1 = ordinal_err(s.thresholds, e1, (int)__shfl_sync(kFull, r.res, j + 1));
            // a last rating without a second: no update and no decay from it
            e1 = two ? e1 : 0.0f;
            const float a2 = two ? a1 : 1.0f;
            // each row's change is summed first and rounded into the row once
            {
                V t = q;
                t.scale(two ? da2 : da);
                t.fma(-p.lr_i * a2 * e0, x0);
                t.fma(-p.lr_i * e1, x1);
                q.add(t);
            }
            {
                V t = g0;
                t.scale(same ? df2 : df);
                t.fma(-p.lr_iqf * (same ? f1 : 1.0f) * e0, x0);
                if (same) t.fma(-p.lr_iqf * e1, x1);
                g0.add(t);
                g0.store(r0, lane);
            }
            if (two && !same) {
                V t = g1;
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
    q.store_cg(s.ifeat + (size_t)i * Fs, lane);
    if (lane == 0) s.ibias[i] = ib;
    if (lane < (int)T) s.bit_bin[(size_t)i * T + lane] = bt0;
    if (lane + 32 < (int)T) s.bit_bin[(size_t)i * T + 32 + lane] = bt1;
    if (lane < (int)NF) s.ibias_freq[(size_t)i * NF + lane] = bf0;
    if (lane + 32 < (int)NF) s.ibias_freq[(size_t)i * NF + 32 + lane] = bf1;
}

// The rest of the items, light ones all: this warp's share of them, k its first.
template <int VPL, bool BF>
__device__ __forceinline__ void light_items(const DeviceState& s, const EpochParams& p, const Bf16Copies& bf, uint32_t k,
                                            int lane, float* ring) {
    while (k < s.n_item_work) {
        const uint32_t i = s.item_work[k];
        if (s.item_off[i] == s.item_off[i + 1]) break;  // no ratings, and none after it
        item_pairs<VPL, BF>(s, p, bf, i, lane, ring);
        if (lane == 0) k = atomicAdd(&s.counters[2], 1u);
        k = __shfl_sync(kFull, k, 0);
    }
}

// Shared floats that `warps` warps' rings take.
__host__ __device__ constexpr size_t light_smem(int warps, uint32_t Fs) { return (size_t)warps * kLightRows * 2 * Fs; }

// Rows of 160 to 256 columns, FP32 or BF16, without the per-day terms and the
// ordinal head (tsvd_item_tiles.cu).
void launch_item_tiles(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf);

}  // namespace tsvd
