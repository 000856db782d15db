// Feature rows held by a warp as packed FP32 pairs, and the strata's shared pieces.
#pragma once
#include "tsvd_epoch.cuh"

namespace tsvd {

using f32x2 = unsigned long long;  // two FP32 values, the operands of the packed FP32 instructions

__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// A lane's VPL values of a feature row (Row<VPL>'s layout), packed in pairs;
// t is the last value of an odd VPL.
template <int VPL>
struct Vec {
    static constexpr int NP = VPL / 2;
    static constexpr bool kOdd = (VPL & 1) != 0;
    f32x2 p[NP > 0 ? NP : 1];
    float t;

    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = 0ull;
        t = 0.0f;
    }
    __device__ __forceinline__ void from(const float (&x)[VPL]) {
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = pack2(x[2 * k], x[2 * k + 1]);
        if constexpr (kOdd) t = x[VPL - 1];
    }
    __device__ __forceinline__ void to(float (&x)[VPL]) const {
#pragma unroll
        for (int k = 0; k < NP; ++k) unpack2(p[k], x[2 * k], x[2 * k + 1]);
        if constexpr (kOdd) x[VPL - 1] = t;
    }
    // rows that no thread writes during the kernel
    __device__ __forceinline__ void load_nc(const float* row, int lane) {
        if constexpr (VPL % 4 == 0) {
#pragma unroll
            for (int c = 0; c < VPL / 4; ++c) {
                const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(row + c * 128 + lane * 4));
                p[2 * c] = v.x;
                p[2 * c + 1] = v.y;
            }
        } else {
            float x[VPL];
            Row<VPL>::load_nc(row, lane, x);
            from(x);
        }
    }
    // rows that other kernels write, through L2
    __device__ __forceinline__ void load_cg(const float* row, int lane) {
        float x[VPL];
        Row<VPL>::load_cg(row, lane, x);
        from(x);
    }
    __device__ __forceinline__ void store_cg(float* row, int lane) const {
        float x[VPL];
        to(x);
        Row<VPL>::store(row, lane, x);
    }
    __device__ __forceinline__ void divide(float d) {
        float x[VPL];
        to(x);
#pragma unroll
        for (int v = 0; v < VPL; ++v) x[v] = x[v] / d;
        from(x);
    }
    __device__ __forceinline__ void load_bf16(const __nv_bfloat16* row, int lane) {
        float x[VPL];
        row_load_bf16<VPL>(row, lane, x);
        from(x);
    }
    // a row that this kernel reads and writes (shared or global memory)
    __device__ __forceinline__ void load(const float* row, int lane) {
        if constexpr (VPL % 4 == 0) {
#pragma unroll
            for (int c = 0; c < VPL / 4; ++c) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(row + c * 128 + lane * 4);
                p[2 * c] = v.x;
                p[2 * c + 1] = v.y;
            }
        } else if constexpr (VPL == 2) {
            p[0] = *reinterpret_cast<const f32x2*>(row + lane * 2);
        } else {
            float x[VPL];
#pragma unroll
            for (int v = 0; v < VPL; ++v) x[v] = row[v * 32 + lane];
            from(x);
        }
    }
    __device__ __forceinline__ void store(float* row, int lane) const {
        if constexpr (VPL % 4 == 0) {
#pragma unroll
            for (int c = 0; c < VPL / 4; ++c)
                *reinterpret_cast<ulonglong2*>(row + c * 128 + lane * 4) = make_ulonglong2(p[2 * c], p[2 * c + 1]);
        } else if constexpr (VPL == 2) {
            *reinterpret_cast<f32x2*>(row + lane * 2) = p[0];
        } else {
            float x[VPL];
            to(x);
#pragma unroll
            for (int v = 0; v < VPL; ++v) row[v * 32 + lane] = x[v];
        }
    }
    __device__ __forceinline__ void scale(float a) {
        const f32x2 aa = pack2(a, a);
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = mul2(aa, p[k]);
        if constexpr (kOdd) t *= a;
    }
    // this += a x
    __device__ __forceinline__ void fma(float a, const Vec& x) {
        const f32x2 aa = pack2(a, a);
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = fma2(aa, x.p[k], p[k]);
        if constexpr (kOdd) t = fmaf(a, x.t, t);
    }
    __device__ __forceinline__ void add(const Vec& x) {
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = add2(p[k], x.p[k]);
        if constexpr (kOdd) t += x.t;
    }
    // this lane's part of the dot product
    __device__ __forceinline__ float dot(const Vec& x) const {
        float r = 0.0f;
        if constexpr (NP > 0) {
            f32x2 acc = mul2(p[0], x.p[0]);
#pragma unroll
            for (int k = 1; k < NP; ++k) acc = fma2(p[k], x.p[k], acc);
            float a, b;
            unpack2(acc, a, b);
            r = a + b;
            if constexpr (kOdd) r = fmaf(t, x.t, r);
        } else {
            r = t * x.t;
        }
        return r;
    }
};

// su += y_j (and sub += b_j, when yb is given) for the items item_of(0 .. n-1),
// added in order: rows of the table y, or of its BF16 copy. kRows rows are asked
// for together; the loop over whole groups has no bounds checks, so a row costs
// its loads, its adds and four instructions more.
template <int VPL, bool BF, class ItemOf>
__device__ __forceinline__ void sum_rows(const float* __restrict__ y, const __nv_bfloat16* __restrict__ ybf,
                                         const float* __restrict__ yb, uint32_t Fs, uint64_t n, ItemOf item_of, int lane,
                                         Vec<VPL>& su, float& sub) {
    constexpr int kRows = VPL >= 5 ? 8 : VPL >= 2 ? 16 : 32;
    auto row = [&](uint32_t it, Vec<VPL>& x) {
        if constexpr (BF) x.load_bf16(ybf + (size_t)it * Fs, lane);
        else x.load_nc(y + (size_t)it * Fs, lane);
    };
    // a chunk's 32 items, one per lane, a chunk ahead
    uint32_t next = (uint64_t)lane < n ? item_of(lane) : 0u;
    for (uint64_t base = 0; base < n; base += 32) {
        const uint32_t cnt = (uint32_t)(n - base < 32 ? n - base : 32);
        const uint32_t mine = next;
        const float b = yb ? __ldg(yb + mine) : 0.0f;
        if (base + 32 + lane < n) next = item_of(base + 32 + lane);
        uint32_t j = 0;
#pragma unroll 1
        for (; j + kRows <= cnt; j += kRows) {
            Vec<VPL> x[kRows];
#pragma unroll
            for (int q = 0; q < kRows; ++q) row(__shfl_sync(kFull, mine, j + q), x[q]);
#pragma unroll
            for (int q = 0; q < kRows; ++q) {
                su.add(x[q]);
                sub += __shfl_sync(kFull, b, j + q);
            }
        }
        if (kRows > 4) {
#pragma unroll 1
            for (; j + 4 <= cnt; j += 4) {
                Vec<VPL> x[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) row(__shfl_sync(kFull, mine, j + q), x[q]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    su.add(x[q]);
                    sub += __shfl_sync(kFull, b, j + q);
                }
            }
        }
#pragma unroll 1
        for (; j < cnt; ++j) {
            Vec<VPL> x;
            row(__shfl_sync(kFull, mine, j), x);
            su.add(x);
            sub += __shfl_sync(kFull, b, j);
        }
    }
}

// The ordinal head's thresholds (lane-uniform); lr_t = 0 in every stratified
// epoch, so they are constant within it.
__device__ __forceinline__ void load_thresholds(const DeviceState& s, float (&th)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) th[k] = s.raw ? __ldg(s.thresholds + k) : 0.0f;
}

// The head's gradient at a score, out of line where the plain chain's loop should
// stay short.
static __device__ __noinline__ float ordinal_err(const float* thresholds, float score, int y) {
    float th[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) th[k] = __ldg(thresholds + k);
    return ordinal_grad(th, score, y);
}

// User-side scalars of one by-item rating: bu_t and cu_t (src/tsvdx4p.rs:690-708).
__device__ __forceinline__ void user_scalars(const DeviceState& s, const Rec& r, float& bu_t, float& cu_t) {
    const uint32_t u = rec_id(r.key), tb = rec_tbin(r.key);
    const bool hud = r.ud < s.n_ud;
    bu_t = __ldg(s.ubias + u) + __ldg(s.but_bin + (size_t)u * s.T + tb) + __ldg(s.alpha_u + u) * r.dev +
           (hud ? __ldg(s.ubias_day + r.ud) : 0.0f) + __ldg(s.ycache_bias + u);
    cu_t = __ldg(s.cu + u) + (hud ? __ldg(s.cut + r.ud) : 0.0f);
}

// The user stratum without the per-day terms, rows up to 256 columns
// (tsvd_user.cu): the n users of `work`, item rows from qe0.
void launch_user_stratum(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf,
                         const uint32_t* work, uint32_t n);

// With the per-day terms (low_memory = false), rows up to 256 columns.
void launch_user_days(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n);

// Rows of more than 256 columns, by a block per user or item (tsvd_wide.cu), where
// wide_pairs_fit(Fs).
bool wide_pairs_fit(uint32_t Fs);
void launch_user_wide_pairs(tsvd_model* m, const DeviceState& s, const EpochParams& p, const uint32_t* work, uint32_t n);
void launch_item_wide_pairs(tsvd_model* m, const DeviceState& s, const EpochParams& p);

// The item stratum of rows up to 256 columns (tsvd_item.cu): the items of
// s.item_work, heaviest first.
void launch_item_stratum(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf);

}  // namespace tsvd
