// Item stratum (fit_epoch_item, src/tsvdx4p.rs:644-762) for rows of 160 to 256
// columns, FP32 or BF16, without the per-day terms and the ordinal head. Narrower
// rows, and those two, take tsvd_item.cu.
#include <algorithm>

#include "tsvd_item.cuh"

namespace tsvd {
namespace {

// ---------------------------------------------------------------------------
// Item stratum. An item's ratings form a serial chain (every update feeds the
// next dot product), and the most-rated items carry ~0.5% of all ratings
// each, so the chain of the hottest item bounds the pass. Items with at least
// s.heavy_min ratings get a whole CTA of kCW + kPW warps, in rounds of kRound ratings:
//   producers (kPW warps) gather the next round's user rows into
//     pe = (p_u + ycache_u) + dev * p2_u plus the rating's bias scalars,
//     form the round's Gram matrix on the tensor cores and from it the
//     round's lower-triangular system (everything about the round that does
//     not depend on the item's current rows);
//   consumers (kCW warps, each owning every kCW-th 32-column stripe of q and
//     of the q^f rows) take the dots with the item's rows, warp 0 solves the
//     system for the round's errors, and all of them apply the closed-form
//     updates to their stripes.
// Rounds are double-buffered with one __syncthreads per round. Lighter items
// take one warp each, with the next rating's rows prefetched into registers.
// ---------------------------------------------------------------------------
constexpr int kRound = 32;  // ratings per buffered round
constexpr uint32_t kMS = kRound + 1;  // padded row stride of the round's system M
constexpr int kCW = 4;                // consumer warps
constexpr int kPW = 8;                // producer warps
constexpr int kItemThreads = (kCW + kPW) * 32;
constexpr int kVecs = 10;             // per-rating vectors of a round
// 16-bit rows of the Gram operands: Fs values + 16 bytes, so that the eight
// 16-byte row segments an ldmatrix reads fall in distinct bank groups
__host__ __device__ constexpr uint32_t hl_pitch(uint32_t Fs) { return Fs * 2 + 16; }
static_assert(kPW * 4 == kRound, "each producer warp stages four of the round's ratings");

// Shared-memory layout of the item pass, in floats (every offset a multiple of 4).
struct ItemSmem {
    uint32_t qfs, qsh, buf, hl, mbuf, vec, pd, sv, ap, st, pw, total;
};
__host__ __device__ inline ItemSmem item_smem(uint32_t Fs, uint32_t NF) {
    ItemSmem L;
    uint32_t o = 0;
    L.qfs = o;  o += NF * (Fs + 4);             // the item's q^f rows, padded
    L.qsh = o;  o += Fs;                        // q at the round's start
    L.buf = o;  o += 2 * kRound * (Fs + 4);     // two rounds of pe rows + {bu_t, cu_t, res, key}
    L.hl = o;   o += 2 * kRound * (Fs / 2 + 4); // high and low parts of the produced round's pe rows
    L.mbuf = o; o += 2 * kRound * kMS;          // two rounds of the system M (row j: M_j,i)
    L.vec = o;  o += 2 * kVecs * kRound;        // two rounds of per-rating weights
    L.pd = o;   o += kCW * 2 * kRound;          // consumers' partial dots
    L.sv = o;   o += 4 * kRound;                // the round's update weights (q, q^f, biases)
    L.ap = o;   o += 4 * kRound;                // per rating {w_q, w_f, decay, bin | previous << 8}
    L.st = o;   o += 132;                       // the item's biases: ib, bit_bin[64], ibias_freq[64]
    L.pw = o;   o += 8 * 36;                    // a_i^n, a_f^n, a_i^n - 1, a_f^n - 1 for n = 0..kRound; rounded a
    L.total = o;
    return L;
}

// The user-side rows of a by-item rating: p_u + ycache_u and p2_u.
template <int VPL, bool BF>
__device__ __forceinline__ void pe_rows(const DeviceState& s, const Bf16Copies& bf, uint32_t u, int lane,
                                        float (&pyc)[VPL], float (&p2)[VPL]) {
    if constexpr (BF) {
        row_load_bf16<VPL>(bf.pyc + (size_t)u * s.Fs, lane, pyc);
        row_load_bf16<VPL>(bf.ufeat2 + (size_t)u * s.Fs, lane, p2);
    } else {
        Row<VPL>::load_nc(s.pyc + (size_t)u * s.Fs, lane, pyc);
        Row<VPL>::load_nc(s.ufeat2 + (size_t)u * s.Fs, lane, p2);
    }
}

// One SGD step of the item chain; qf_at(v) is this lane's v-th element of q^f[fb].
template <int VPL, class QF>
__device__ __forceinline__ void item_step(const DeviceState& s, const EpochParams& p, float gb, float (&q)[VPL],
                                          QF&& qf_at, const float (&pe)[VPL], float bu_t, float cu_t, float res,
                                          uint32_t tb, uint32_t fb, int lane, ItemState& st) {
    const float bit = __shfl_sync(kFull, tb < 32 ? st.bt0 : st.bt1, tb & 31);
    const float ibf = __shfl_sync(kFull, fb < 32 ? st.bf0 : st.bf1, fb & 31);
    const float bi_t = st.ib + bit + ibf;
    float qfv[VPL], part = 0.0f;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        qfv[v] = qf_at(v);
        part += pe[v] * (q[v] + qfv[v]);
    }
    const float dot = warp_sum(part);
    const float err = (gb + bu_t + bi_t * cu_t + dot) - res;
    const float ec = err * cu_t;
    st.ib -= p.lr_ib * ec;
    const float nb = bit - p.lr_ti * ec;
    if (lane == (int)(tb & 31)) {
        if (tb < 32) st.bt0 = nb;
        else st.bt1 = nb;
    }
    const float nf = ibf - p.lr_ibf * ec;
    if (lane == (int)(fb & 31)) {
        if (fb < 32) st.bf0 = nf;
        else st.bf1 = nf;
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        const float qi = q[v];
        q[v] = qi - p.lr_i * (err * pe[v] + p.reg_i * qi);
        qfv[v] = qfv[v] - p.lr_iqf * (err * pe[v] + p.reg_iqf * qfv[v]);
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v) qf_at(v) = qfv[v];
}

// One light item by one warp, one rating at a time (fit_epoch_item,
// src/tsvdx4p.rs:644-762), the next one's rows loaded a step ahead. (Two at a
// time as in tsvd_item.cuh has a chain half as long, but its q^f rows miss what L1
// is left beside the heavy items' shared memory: 100,480,507 ratings, f = 256,
// 69.9 against 60.4 ms.)
template <int VPL, bool BF>
__device__ void item_light(const DeviceState& s, const EpochParams& p, const Bf16Copies& bf, uint32_t i, int lane) {
    const uint32_t Fs = s.Fs, NF = s.NF;
    const uint64_t a = s.item_off[i], b = s.item_off[i + 1];
    if (a == b) return;
    float q[VPL];
    Row<VPL>::load_cg(s.ifeat + (size_t)i * Fs, lane, q);
    ItemState st = load_item_state(s, i, lane);
    float* qf_base = s.ifeat_freq + (size_t)i * NF * Fs;
    const float gb = s.gbias;
    for (uint64_t base = a; base < b; base += 32) {
        const uint32_t cnt = (uint32_t)(b - base < 32 ? b - base : 32);
        // the chunk's records and user-side scalars, one rating per lane
        Rec mine{};
        float bu_l = 0.0f, cu_l = 0.0f;
        if (lane < (int)cnt) {
            mine = load_rec(s.irec + base + lane);
            user_scalars(s, mine, bu_l, cu_l);
        }
        float pn[VPL], p2n[VPL];
        auto fetch = [&](uint32_t j) {
            const uint32_t uj = rec_id(__shfl_sync(kFull, mine.key, j));
            pe_rows<VPL, BF>(s, bf, uj, lane, pn, p2n);
        };
        fetch(0);
        // the q^f row of the current rating's bin; the next rating's row is
        // loaded a step ahead when its bin differs (this rating leaves it alone)
        uint32_t fcur = rec_fbin(__shfl_sync(kFull, mine.key, 0));
        float qfv[VPL];
        Row<VPL>::load_cg(qf_base + (size_t)fcur * Fs, lane, qfv);
        for (uint32_t j = 0; j < cnt; ++j) {
            const Rec r = shfl_rec(mine, j);
            float pe[VPL];
#pragma unroll
            for (int v = 0; v < VPL; ++v) pe[v] = pn[v] + r.dev * p2n[v];
            if (j + 1 < cnt) fetch(j + 1);
            const float bu_t = __shfl_sync(kFull, bu_l, j), cu_t = __shfl_sync(kFull, cu_l, j);
            const uint32_t tb = rec_tbin(r.key), fb = fcur;
            const uint32_t fnext = j + 1 < cnt ? rec_fbin(__shfl_sync(kFull, mine.key, j + 1)) : fcur;
            float qfn[VPL];
            if (fnext != fcur) Row<VPL>::load_cg(qf_base + (size_t)fnext * Fs, lane, qfn);
            item_step<VPL>(s, p, gb, q, [&](int v) -> float& { return qfv[v]; }, pe, bu_t, cu_t, r.res, tb, fb,
                           lane, st);
            Row<VPL>::store(qf_base + (size_t)fcur * Fs, lane, qfv);
            if (fnext != fcur) {
#pragma unroll
                for (int v = 0; v < VPL; ++v) qfv[v] = qfn[v];
            }
            fcur = fnext;
        }
    }
    Row<VPL>::store(s.ifeat + (size_t)i * Fs, lane, q);
    store_item_state(s, i, lane, st);
}

// Packed BF16 pairs of (x, y): the values rounded, and what that leaves rounded.
__device__ __forceinline__ void split_pair_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 f = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// d (16x8, FP32) += a (16x16, row-major) . b (16x8, column-major), of FP16 or BF16
template <bool BP>
__device__ __forceinline__ void mma_parts(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (BP)
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else mma_f16(d, a, b0, b1);
}

// One staged rating: its FP32 pe row (for the consumers) and the high and low parts
// of it (the Gram operands), each element split once: FP16 parts, scaled, and the
// inverse of the scale is returned, or with `BP` BF16 parts.
template <int VPL, bool BP>
__device__ __forceinline__ float stage_row(float* row, uint8_t* hi_row, uint8_t* lo_row, int lane,
                                           const float (&pe)[VPL]) {
    float unscale = 1.0f, sc = 1.0f;
    if constexpr (!BP) {
        unscale = row_unscale(pe);
        sc = row_scale(unscale);
    }
    auto split = [&](float x, float y, uint32_t& h, uint32_t& l) {
        if constexpr (BP) split_pair_bf16(x, y, h, l);
        else split_pair(x * sc, y * sc, h, l);
    };
    if constexpr (VPL % 4 == 0) {
#pragma unroll
        for (int c = 0; c < VPL / 4; ++c) {
            const int col = c * 128 + lane * 4;
            const float4 x = make_float4(pe[4 * c], pe[4 * c + 1], pe[4 * c + 2], pe[4 * c + 3]);
            *reinterpret_cast<float4*>(row + col) = x;
            uint2 h, l;
            split(x.x, x.y, h.x, l.x);
            split(x.z, x.w, h.y, l.y);
            *reinterpret_cast<uint2*>(hi_row + 2 * col) = h;
            *reinterpret_cast<uint2*>(lo_row + 2 * col) = l;
        }
    } else {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            const int col = Row<VPL>::elem(lane, v);
            row[col] = pe[v];
            uint32_t h, l;
            split(pe[v], 0.0f, h, l);
            reinterpret_cast<uint16_t*>(hi_row)[col] = (uint16_t)h;
            reinterpret_cast<uint16_t*>(lo_row)[col] = (uint16_t)l;
        }
    }
    return unscale;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// BP: the rounds' dots from BF16 parts (launch_form).
template <int VPL, bool BF, bool BP>
__global__ void __launch_bounds__(kItemThreads, 1) k_item_pass(DeviceState s, EpochParams p, Bf16Copies bf) {
    extern __shared__ __align__(16) float smem[];
    __shared__ uint32_t sh_k;
    static_assert(kCW == 4, "the consumers' partial dots are summed as (0 + 1) + (2 + 3)");
    constexpr int CPL = (VPL + kCW - 1) / kCW;  // 32-column stripes per consumer warp
    constexpr int kChunk = 8;                   // ratings per step of the consumers' apply
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t Fs = s.Fs, NF = s.NF, T = s.T, NS = Fs / 32;
    const uint32_t stride = Fs + 4;  // one staged rating: pe row + {bu_t, cu_t, res, key}
    const uint32_t qs = Fs + 4;      // padded q^f row stride
    const ItemSmem L = item_smem(Fs, NF);
    float* qfs = smem + L.qfs;
    float* qsh = smem + L.qsh;
    float* buf = smem + L.buf;
    uint8_t* hl = reinterpret_cast<uint8_t*>(smem + L.hl);
    const uint32_t hp = hl_pitch(Fs);
    float* mbuf = smem + L.mbuf;
    float* vec = smem + L.vec;
    float* pd = smem + L.pd;
    float* sv = smem + L.sv;
    float4* ap = reinterpret_cast<float4*>(smem + L.ap);
    float* sst = smem + L.st;
    if (threadIdx.x < 2) decay_powers<kRound>(smem + L.pw + threadIdx.x * 144, p, threadIdx.x == 1);
    const float gb = s.gbias;
    for (;;) {
        if (threadIdx.x == 0) sh_k = atomicAdd(&s.counters[2], 1u);
        __syncthreads();
        const uint32_t k = sh_k;
        __syncthreads();
        if (k >= s.n_item_work) return;
        const uint32_t i = s.item_work[k];
        const uint64_t a = s.item_off[i], b = s.item_off[i + 1];
        if (b - a < s.heavy_min) {
            // Items are ordered heaviest first: from here on every item is light.
            if (warp == 0) item_light<VPL, BF>(s, p, bf, i, lane);
            for (;;) {
                uint32_t k2 = 0;
                if (lane == 0) k2 = atomicAdd(&s.counters[2], 1u);
                k2 = __shfl_sync(kFull, k2, 0);
                if (k2 >= s.n_item_work) return;
                item_light<VPL, BF>(s, p, bf, s.item_work[k2], lane);
            }
        }
        // ---------------- heavy item: whole CTA ----------------
        for (uint32_t e = threadIdx.x; e < NF * Fs; e += blockDim.x)
            qfs[(e / Fs) * qs + e % Fs] = __ldcg(s.ifeat_freq + (size_t)i * NF * Fs + e);
        const uint64_t n = b - a;
        const float* apow = smem + L.pw + (n >= s.rounded_decay_min ? 144 : 0);
        const float *fpow = apow + 36, *adec = apow + 72, *fdec = apow + 108;
        const uint32_t rounds = (uint32_t)((n + kRound - 1) / kRound);
        if (threadIdx.x < 64) {
            const uint32_t t = threadIdx.x;
            if (t == 0) sst[0] = __ldcg(s.ibias + i);
            sst[1 + t] = t < T ? __ldcg(s.bit_bin + (size_t)i * T + t) : 0.0f;
            sst[65 + t] = t < NF ? __ldcg(s.ibias_freq + (size_t)i * NF + t) : 0.0f;
        }
        float qv[CPL];  // consumer warp c: q columns 32 (c + kCW t) + lane
        if (warp < kCW) {
#pragma unroll
            for (int t = 0; t < CPL; ++t) {
                const uint32_t sc = warp + kCW * t;
                qv[t] = sc < NS ? __ldcg(s.ifeat + (size_t)i * Fs + 32 * sc + lane) : 0.0f;
            }
        }
        auto round_len = [&](uint32_t r) -> uint32_t {
            const uint64_t left = n - (uint64_t)r * kRound;
            return (uint32_t)(left < (uint64_t)kRound ? left : (uint64_t)kRound);
        };
        // Producers load records two rounds ahead (one per lane) and the next
        // round's user scalars (on the lanes that stage them) a round ahead,
        // so that their latency overlaps the wait for the consumers.
        Rec rc1{}, rc2{};
        float us[7] = {};  // ubias, but_bin, alpha_u, ubias_day, ycache_bias, cu, cut
        // user rows (p_u + ycache_u, p2_u) of ratings pw and pw + 8 of the next
        // round, loaded at the end of the previous producer phase
        float px0[VPL], py0[VPL], px1[VPL], py1[VPL];
        auto fetch_rows0 = [&](uint32_t r) {  // rc1 holds round r's records
            const int pw = warp - kCW;
            const uint32_t m = round_len(r), j0 = pw, j1 = pw + kPW;
            const uint32_t u0 = rec_id(__shfl_sync(kFull, rc1.key, j0));
            const uint32_t u1 = rec_id(__shfl_sync(kFull, rc1.key, j1));
#pragma unroll
            for (int v = 0; v < VPL; ++v) px0[v] = py0[v] = px1[v] = py1[v] = 0.0f;
            if (j0 < m) pe_rows<VPL, BF>(s, bf, u0, lane, px0, py0);
            if (j1 < m) pe_rows<VPL, BF>(s, bf, u1, lane, px1, py1);
        };
        auto fetch_records = [&](uint32_t r, Rec& out) {
            out = Rec{};
            if (r < rounds && lane < (int)round_len(r)) out = load_rec(s.irec + a + (uint64_t)r * kRound + lane);
        };
        auto fetch_scalars = [&](uint32_t r) {  // rc1 holds round r's records
            const int pw = warp - kCW;
            if (lane < (int)round_len(r) && (lane & (kPW - 1)) == pw) {
                const uint32_t u = rec_id(rc1.key), tb = rec_tbin(rc1.key);
                const bool hud = rc1.ud < s.n_ud;
                us[0] = __ldg(s.ubias + u);
                us[1] = __ldg(s.but_bin + (size_t)u * s.T + tb);
                us[2] = __ldg(s.alpha_u + u);
                us[3] = hud ? __ldg(s.ubias_day + rc1.ud) : 0.0f;
                us[4] = __ldg(s.ycache_bias + u);
                us[5] = __ldg(s.cu + u);
                us[6] = hud ? __ldg(s.cut + rc1.ud) : 0.0f;
            }
        };
        // Producer warp pw: round r's pe rows pw, pw + 8, pw + 16, pw + 24 and
        // their scalars, then (pw < 6) a Gram tile and the entries of the
        // round's system M that it holds, or (pw == 6) the per-rating weights.
        auto produce = [&](uint32_t r) {
            const int pw = warp - kCW;
            float* dst = buf + (size_t)(r & 1) * kRound * stride;
            float* Mb = mbuf + (size_t)(r & 1) * kRound * kMS;
            float* V = vec + (size_t)(r & 1) * kVecs * kRound;
            const uint32_t m = round_len(r);
            const bool valid = lane < (int)m;
            const Rec mine = rc1;
            if ((lane & (kPW - 1)) == pw) {
                // bu_t, cu_t as user_scalars forms them (src/tsvdx4p.rs:690-708)
                const float bu = valid ? us[0] + us[1] + us[2] * mine.dev + us[3] + us[4] : 0.0f;
                const float cu = valid ? us[5] + us[6] : 0.0f;
                float* row = dst + (size_t)lane * stride;
                row[Fs] = bu;
                row[Fs + 1] = cu;
                row[Fs + 2] = mine.res;
                row[Fs + 3] = __uint_as_float(mine.key);
            }
            // ratings pw + 16 and pw + 24: their user rows are loaded now, while
            // ratings pw and pw + 8 (loaded a phase earlier) are staged; rows
            // m..31 of a partial round are zero
            {
                const uint32_t j2 = pw + 16, j3 = pw + 24;
                const uint32_t u2 = rec_id(__shfl_sync(kFull, mine.key, j2));
                const uint32_t u3 = rec_id(__shfl_sync(kFull, mine.key, j3));
                float x2[VPL], y2[VPL], x3[VPL], y3[VPL];
#pragma unroll
                for (int v = 0; v < VPL; ++v) x2[v] = y2[v] = x3[v] = y3[v] = 0.0f;
                if (j2 < m) pe_rows<VPL, BF>(s, bf, u2, lane, x2, y2);
                if (j3 < m) pe_rows<VPL, BF>(s, bf, u3, lane, x3, y3);
                const uint32_t j0 = pw, j1 = pw + kPW;
                const float d0 = __shfl_sync(kFull, mine.dev, j0), d1 = __shfl_sync(kFull, mine.dev, j1);
                const float d2 = __shfl_sync(kFull, mine.dev, j2), d3 = __shfl_sync(kFull, mine.dev, j3);
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    px0[v] = px0[v] + d0 * py0[v];
                    px1[v] = px1[v] + d1 * py1[v];
                }
                const float s0 = stage_row<VPL, BP>(dst + (size_t)j0 * stride, hl + (size_t)j0 * hp,
                                                 hl + (size_t)(kRound + j0) * hp, lane, px0);
                const float s1 = stage_row<VPL, BP>(dst + (size_t)j1 * stride, hl + (size_t)j1 * hp,
                                                 hl + (size_t)(kRound + j1) * hp, lane, px1);
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    x2[v] = x2[v] + d2 * y2[v];
                    x3[v] = x3[v] + d3 * y3[v];
                }
                const float s2 = stage_row<VPL, BP>(dst + (size_t)j2 * stride, hl + (size_t)j2 * hp,
                                                 hl + (size_t)(kRound + j2) * hp, lane, x2);
                const float s3 = stage_row<VPL, BP>(dst + (size_t)j3 * stride, hl + (size_t)j3 * hp,
                                                 hl + (size_t)(kRound + j3) * hp, lane, x3);
                if (!BP && lane < 4) V[9 * kRound + pw + kPW * lane] = lane == 0 ? s0 : lane == 1 ? s1 : lane == 2 ? s2 : s3;
            }
            // all rows of the round are in place before the Gram products
            asm volatile("bar.sync 2, %0;" ::"r"(kPW * 32) : "memory");
            const uint32_t fbl = rec_fbin(mine.key);
            // the round's ratings of each frequency bin (valid ratings only)
            const unsigned same = __match_any_sync(kFull, valid ? fbl : 64u + (uint32_t)lane);
            if (pw < 6) {
                // G = PE PE^T on the tensor cores, from the rows' high and low parts.
                // Tile pw of the six 16x8 tiles (rows x columns) that hold
                // every pair row < column.
                const int mt = pw < 4 ? 0 : 1, nt = pw < 4 ? pw : pw - 2;
                const int gid = lane >> 2, tig = lane & 3;
                // ldmatrix row addresses: A (16x16) as four 8x8 matrices
                // (rows 0-7 | 8-15) x (k 0-7 | 8-15); B's high and low parts
                // (8 pe rows x k 0-7 | 8-15) in one x4
                const uint32_t hl_s = smem_u32(hl);
                const int ar = mt * 16 + (lane & 7) + 8 * ((lane >> 3) & 1), ak = 8 * (lane >> 4);
                const uint32_t a_hi = hl_s + (uint32_t)(ar * hp + 2 * ak);
                const uint32_t a_lo = a_hi + (uint32_t)(kRound * hp);
                const int br = nt * 8 + (lane & 7), bk = 8 * ((lane >> 3) & 1);
                const uint32_t b_hl = hl_s + (uint32_t)(((lane >> 4) * kRound + br) * hp + 2 * bk);
                float d[6][4] = {};
#pragma unroll 2
                for (uint32_t k0 = 0; k0 < Fs; k0 += 32) {
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const uint32_t kb = 2 * (k0 + 16 * hh);
                        uint32_t ah[4], al[4], bb[4];
                        ldmatrix_x4(ah, a_hi + kb);
                        ldmatrix_x4(al, a_lo + kb);
                        ldmatrix_x4(bb, b_hl + kb);
                        mma_parts<BP>(d[3 * hh], al, bb[0], bb[1]);
                        mma_parts<BP>(d[3 * hh + 1], ah, bb[2], bb[3]);
                        mma_parts<BP>(d[3 * hh + 2], ah, bb[0], bb[1]);
                    }
                }
                // The round's errors solve err = C - M err with M unit lower
                // triangular: M_ji (i < j) is the effect of err_i on rating j
                // through q (a_i^(j-1-i) G_ij), the q^f row of a shared bin
                // (a_f^(same-bin ratings between) G_ij) and the item biases.
                // This lane's four entries (i, j) give M_ji and M_ij = 0.
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int ii = mt * 16 + gid + 8 * (e >> 1), jj = nt * 8 + 2 * tig + (e & 1);
                    const uint32_t ki = __shfl_sync(kFull, mine.key, ii), kj = __shfl_sync(kFull, mine.key, jj);
                    const unsigned samej = __shfl_sync(kFull, same, jj);
                    if (ii < jj) {
                        float v = 0.0f;
                        if (jj < (int)m) {
                            float g = ((d[0][e] + d[1][e]) + (d[3][e] + d[4][e])) + (d[2][e] + d[5][e]);
                            if constexpr (!BP) g = g * V[9 * kRound + ii] * V[9 * kRound + jj];
                            const float cui = dst[(size_t)ii * stride + Fs + 1], cuj = dst[(size_t)jj * stride + Fs + 1];
                            const bool same_f = rec_fbin(ki) == rec_fbin(kj), same_t = rec_tbin(ki) == rec_tbin(kj);
                            const float bias_lr = p.lr_ib + (same_t ? p.lr_ti : 0.0f) + (same_f ? p.lr_ibf : 0.0f);
                            const unsigned between = ((1u << jj) - 1u) & ~((2u << ii) - 1u);
                            v = cuj * cui * bias_lr + p.lr_i * apow[jj - 1 - ii] * g +
                                (same_f ? p.lr_iqf * fpow[__popc(samej & between)] * g : 0.0f);
                        }
                        Mb[(size_t)jj * kMS + ii] = v;
                        Mb[(size_t)ii * kMS + jj] = 0.0f;
                    } else if (ii == jj) {
                        Mb[(size_t)ii * kMS + ii] = 0.0f;
                    }
                }
            } else if (pw == 6) {
                // per-rating weights of the round (j = lane)
                const unsigned below = (1u << lane) - 1u, above = ~((2u << lane) - 1u);
                const unsigned earlier = same & below;
                V[lane] = apow[lane];                                       // a_i^j
                V[kRound + lane] = fpow[__popc(earlier)];                   // a_f^(earlier ratings of the bin)
                V[2 * kRound + lane] = valid ? apow[valid ? m - 1 - lane : 0] : 0.0f;  // a_i^(m-1-j)
                V[3 * kRound + lane] = fpow[__popc(same & above)];          // a_f^(later ratings of the bin)
                // the first rating of a bin applies the decay of all its ratings to the bin's row (less one)
                V[4 * kRound + lane] = (valid && earlier == 0u) ? fdec[__popc(same)] : 0.0f;
                V[5 * kRound + lane] = __uint_as_float(fbl);
                if (lane == 0) V[6 * kRound] = adec[m];                     // a_i^m - 1
                // the previous rating of the same bin in the round, or -1
                V[7 * kRound + lane] = __int_as_float(earlier ? 31 - __clz((int)earlier) : -1);
                V[8 * kRound + lane] = __uint_as_float(rec_tbin(mine.key));
            }
            // the next rounds' loads
            rc1 = rc2;
            if (r + 1 < rounds) {
                fetch_scalars(r + 1);
                fetch_rows0(r + 1);
            }
            fetch_records(r + 2, rc2);
        };
        if (warp >= kCW) {
            fetch_records(0, rc1);
            fetch_records(1, rc2);
            fetch_scalars(0);
            fetch_rows0(0);
            produce(0);
        }
        __syncthreads();
        for (uint32_t r = 0; r < rounds; ++r) {
            if (warp >= kCW) {
                if (r + 1 < rounds) produce(r + 1);
            } else {
                // Lookahead over the round's m ratings (all of one item): with
                // q_k, qf_k the item rows before rating k, and pe_k fixed in
                // the item stratum,
                //   q_k . pe_k = a_i^k (q_0 . pe_k) - lr_i sum_{j<k} a_i^(k-1-j) err_j G_jk
                // and likewise for the q^f row of pe_k's frequency bin over the
                // earlier ratings of the same bin. The dots with q_0 are taken
                // once per round; the round's updates are applied in closed form,
                //   q_m = a_i^m q_0 - lr_i sum_k a_i^(m-1-k) err_k pe_k.
                const float* src = buf + (size_t)(r & 1) * kRound * stride;
                const float* Mb = mbuf + (size_t)(r & 1) * kRound * kMS;
                const float* V = vec + (size_t)(r & 1) * kVecs * kRound;
                const uint32_t m = round_len(r);
                const float* myrow = src + (size_t)lane * stride;
                const uint32_t keyl = __float_as_uint(myrow[Fs + 3]);
                const uint32_t fbl = rec_fbin(keyl);
                // partial dots of pe_lane with q_0 and q^f_0[fb] over this warp's stripes
#pragma unroll
                for (int t = 0; t < CPL; ++t) {
                    const uint32_t sc = warp + kCW * t;
                    if (sc < NS) qsh[32 * sc + lane] = qv[t];
                }
                __syncwarp();
                {
                    float s0 = 0.0f, s1 = 0.0f, e0 = 0.0f, e1 = 0.0f;
#pragma unroll
                    for (int t = 0; t < CPL; ++t) {
                        const uint32_t sc = warp + kCW * t;
                        if (sc < NS) {
                            const float4* x4 = reinterpret_cast<const float4*>(myrow + 32 * sc);
                            const float4* y4 = reinterpret_cast<const float4*>(qsh + 32 * sc);
                            const float4* z4 = reinterpret_cast<const float4*>(qfs + (size_t)fbl * qs + 32 * sc);
#pragma unroll
                            for (int k4 = 0; k4 < 8; ++k4) {
                                const float4 x = x4[k4], y = y4[k4], z = z4[k4];
                                s0 = fmaf(x.x, y.x, s0);
                                s1 = fmaf(x.y, y.y, s1);
                                s0 = fmaf(x.z, y.z, s0);
                                s1 = fmaf(x.w, y.w, s1);
                                e0 = fmaf(x.x, z.x, e0);
                                e1 = fmaf(x.y, z.y, e1);
                                e0 = fmaf(x.z, z.z, e0);
                                e1 = fmaf(x.w, z.w, e1);
                            }
                        }
                    }
                    pd[(2 * warp) * kRound + lane] = s0 + s1;
                    pd[(2 * warp + 1) * kRound + lane] = e0 + e1;
                }
                asm volatile("bar.sync 1, %0;" ::"r"(kCW * 32) : "memory");
                float wb = 0.0f;
                if (warp == 0) {
                    const float sq = (pd[lane] + pd[2 * kRound + lane]) + (pd[4 * kRound + lane] + pd[6 * kRound + lane]);
                    const float sf =
                        (pd[kRound + lane] + pd[3 * kRound + lane]) + (pd[5 * kRound + lane] + pd[7 * kRound + lane]);
                    const float bu_t = myrow[Fs], cu_t = myrow[Fs + 1], res = myrow[Fs + 2];
                    const uint32_t tb = rec_tbin(keyl);
                    const bool valid = lane < (int)m;
                    const float bi0 = sst[0] + sst[1 + tb] + sst[65 + fbl];
                    float x = ((gb + bu_t + bi0 * cu_t) + (V[lane] * sq + V[kRound + lane] * sf)) - res;
                    x = valid ? x : 0.0f;
                    // Forward substitution in blocks of four: each block's
                    // four values are broadcast at once, every lane solves
                    // the block's 4x4 system, and the lanes past the block
                    // subtract its contributions. M is zero on and above the
                    // diagonal, so the lanes of the block get their own value
                    // and earlier lanes keep theirs.
                    const float* Mr = Mb + (size_t)lane * kMS;
#pragma unroll
                    for (int c = 0; c < kRound; c += 4) {
                        const float s0 = __shfl_sync(kFull, x, c), s1 = __shfl_sync(kFull, x, c + 1);
                        const float s2 = __shfl_sync(kFull, x, c + 2), s3 = __shfl_sync(kFull, x, c + 3);
                        const float* B1 = Mb + (size_t)(c + 1) * kMS + c;
                        const float* B2 = Mb + (size_t)(c + 2) * kMS + c;
                        const float* B3 = Mb + (size_t)(c + 3) * kMS + c;
                        const float e1 = fmaf(-B1[0], s0, s1);
                        const float e2 = fmaf(-B2[1], e1, fmaf(-B2[0], s0, s2));
                        const float e3 = fmaf(-B3[2], e2, fmaf(-B3[1], e1, fmaf(-B3[0], s0, s3)));
                        x = fmaf(-Mr[c + 3], e3, fmaf(-Mr[c + 2], e2, fmaf(-Mr[c + 1], e1, fmaf(-Mr[c], s0, x))));
                    }
                    const float wq = valid ? p.lr_i * V[2 * kRound + lane] * x : 0.0f;
                    const float wf = valid ? p.lr_iqf * V[3 * kRound + lane] * x : 0.0f;
                    const int pv = __float_as_int(V[7 * kRound + lane]);
                    ap[lane] = make_float4(wq, wf, V[4 * kRound + lane], __uint_as_float(fbl | (uint32_t)(pv + 1) << 8));
                    wb = valid ? x * cu_t : 0.0f;
                    sv[2 * kRound + lane] = wb;
                }
                asm volatile("bar.sync 1, %0;" ::"r"(kCW * 32) : "memory");
                // q and q^f stripes, kChunk ratings at a time: the chunk's pe
                // and q^f values are loaded together, a rating whose bin an
                // earlier rating of the chunk updated takes that value from
                // registers, and the chunk's rows are stored at its end.
                if (warp >= 2) {
                    // item biases, beside the warps' own stripes: warp 2 the
                    // item bias and the time-bin biases, warp 3 the
                    // frequency-bin biases
                    if (warp == 2) {
                        const float sw = warp_sum(sv[2 * kRound + lane]);
                        if (lane == 0) sst[0] = sst[0] - p.lr_ib * sw;
                    }
                    const int vo = warp == 2 ? 8 : 5;  // the ratings' bins: tb (vector 8) or fb (vector 5)
                    float d0 = 0.0f, d1 = 0.0f;
#pragma unroll 8
                    for (int c = 0; c < kRound; ++c) {
                        const float e = sv[2 * kRound + c];
                        const uint32_t bk = __float_as_uint(V[vo * kRound + c]);
                        d0 += lane == (int)bk ? e : 0.0f;
                        d1 += lane + 32 == (int)bk ? e : 0.0f;
                    }
                    const float lr = warp == 2 ? p.lr_ti : p.lr_ibf;
                    float* bb = sst + (warp == 2 ? 1 : 65);
                    bb[lane] = bb[lane] - lr * d0;
                    bb[lane + 32] = bb[lane + 32] - lr * d1;
                }
                const float am = V[6 * kRound];
#pragma unroll
                for (int t = 0; t < CPL; ++t) qv[t] = fmaf(am, qv[t], qv[t]);
#pragma unroll 1
                for (int c0 = 0; c0 < kRound; c0 += kChunk) {
                    float pk[kChunk][CPL], ol[kChunk][CPL], nv[kChunk][CPL];
                    float4 w4[kChunk];
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        w4[u] = ap[c0 + u];
                        const uint32_t fk = __float_as_uint(w4[u].w) & 0xffu;
#pragma unroll
                        for (int t = 0; t < CPL; ++t) {
                            const uint32_t sc = warp + kCW * t;
                            pk[u][t] = sc < NS ? src[(size_t)(c0 + u) * stride + 32 * sc + lane] : 0.0f;
                            ol[u][t] = sc < NS ? qfs[(size_t)fk * qs + 32 * sc + lane] : 0.0f;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        const float wq = w4[u].x, wf = w4[u].y, dk = w4[u].z;
                        const int pv = (int)(__float_as_uint(w4[u].w) >> 8) - 1;
#pragma unroll
                        for (int t = 0; t < CPL; ++t) {
                            qv[t] = fmaf(-wq, pk[u][t], qv[t]);
                            float o = ol[u][t];
#pragma unroll
                            for (int u2 = 0; u2 < u; ++u2) o = pv == c0 + u2 ? nv[u2][t] : o;
                            nv[u][t] = fmaf(-wf, pk[u][t], fmaf(dk, o, o));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        // (ratings m..31 of a partial round would store stale rows)
                        if (c0 + u >= (int)m) break;
                        const uint32_t fk = __float_as_uint(w4[u].w) & 0xffu;
#pragma unroll
                        for (int t = 0; t < CPL; ++t) {
                            const uint32_t sc = warp + kCW * t;
                            if (sc < NS) qfs[(size_t)fk * qs + 32 * sc + lane] = nv[u][t];
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (warp < kCW) {
#pragma unroll
            for (int t = 0; t < CPL; ++t) {
                const uint32_t sc = warp + kCW * t;
                if (sc < NS) s.ifeat[(size_t)i * Fs + 32 * sc + lane] = qv[t];
            }
        }
        if (threadIdx.x < 64) {
            const uint32_t t = threadIdx.x;
            if (t == 0) s.ibias[i] = sst[0];
            if (t < T) s.bit_bin[(size_t)i * T + t] = sst[1 + t];
            if (t < NF) s.ibias_freq[(size_t)i * NF + t] = sst[65 + t];
        }
        for (uint32_t e = threadIdx.x; e < NF * Fs; e += blockDim.x)
            __stcg(s.ifeat_freq + (size_t)i * NF * Fs + e, qfs[(e / Fs) * qs + e % Fs]);
        __syncthreads();
    }
}

template <int VPL, bool BF, bool BP>
void launch_tiles(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    auto kern = k_item_pass<VPL, BF, BP>;
    const size_t smem = (size_t)item_smem(s.Fs, s.NF).total * sizeof(float);
    allow_dyn_smem(kern, smem);
    int dev = 0, sms = 0;
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    kern<<<(unsigned)sms, kItemThreads, smem, m->stream>>>(s, p, bf);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

// Items of 32,768 ratings and more have always had their dots from BF16 parts, 16 bits:
// where no smaller item takes a block they keep them (100,480,507 ratings, f = 256:
// item pass 59.2 ms, 62.4 from the FP16 parts that the smaller ones need).
template <int VPL, bool BF>
void launch_form(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    if (s.heavy_min >= s.rounded_decay_min) launch_tiles<VPL, BF, true>(m, s, p, bf);
    else launch_tiles<VPL, BF, false>(m, s, p, bf);
}

template <int VPL>
void launch_rows(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    if (bf.pyc) launch_form<VPL, true>(m, s, p, bf);
    else launch_form<VPL, false>(m, s, p, bf);
}

}  // namespace

void launch_item_tiles(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    switch (s.Fs / 32) {
        case 5: launch_rows<5>(m, s, p, bf); break;
        case 6: launch_rows<6>(m, s, p, bf); break;
        case 7: launch_rows<7>(m, s, p, bf); break;
        case 8: launch_rows<8>(m, s, p, bf); break;
        default: throw Error(TSVD_ERR_UNSUPPORTED, "item tiles take rows of 160 to 256 columns");
    }
}

}  // namespace tsvd
