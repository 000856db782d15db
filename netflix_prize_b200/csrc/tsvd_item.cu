// Item stratum of the stratified schedule (fit_epoch_item,
// src/tsvdx4p.rs:644-762): items in parallel, user tables frozen, each item's
// ratings one after another, kRound at a time.
//
// The opposite rows of an item's ratings, pe_k = (p_u + ycache_u) + dev p2_u
// (with the per-day terms also ufeat_day and ycache_day of the rating's day),
// do not change in this stratum. With x - lr (g + reg x) = a x - lr g for the
// item's row q, and likewise for the q^f row of a rating's frequency bin,
//   q_k . pe_k = a^k (q_0 . pe_k) - lr sum_{i<k} a^(k-1-i) err_i (pe_i . pe_k),
// so the round's errors solve the unit lower triangular system
//   err = C - M err:  C from the rows at the round's start, M from the dots of
// the round's pe rows and the biases' shared bins. With the ordinal head C is a
// score and err its gradient, taken one rating after another.
//
// A CTA takes an item; its warps work on three rounds at once, one step of all
// of them between two CTA barriers:
//   producers (kPW warps), round r + 2: gather the user rows (asked for a step
//     ahead) and write pe, then six of them form the pairs' dots on the tensor
//     cores and M; of the other two, one brings the item's biases past round
//     r - 1 and forms C's bias part of round r, one inverts the two diagonal 16 x
//     16 blocks of I + M of round r + 1 and lays out round r + 3;
//   consumers, round r: each holds some columns of q (registers) and of the q^f
//     rows (shared memory); partial dots, the errors (every warp for itself), and
//     the closed-form updates of its columns. A frequency bin's row takes the sum
//     of its ratings' updates from a table of weights that is zero outside the
//     bin, so all of its inner loops are straight.
// So the serial part of a round is the consumers' alone.
#include <algorithm>

#include "tsvd_item.cuh"

namespace tsvd {
namespace {

// How the user rows are read: FP32, their BF16 copies, or FP32 with the
// per-day rows (low_memory = false).
enum { kPlain = 0, kBf16 = 1, kPerDay = 2 };

constexpr int kRound = 32;  // ratings per round
// Rows from this many 32-column stripes on go to tsvd_item_tiles.cu where it
// takes them: its round is bound by shared-memory traffic that this kernel has
// more of (f = 256, hottest item of 476,450 ratings: 127 against 150 ns a rating).
// Item pass there and here, ms, of 25 M ratings (of 1 M): 256 columns 15.8 and 19.8
// (1.27, 1.50), 224 16.4 and 16.8 (1.28, 1.29), 192 15.4 and 14.0 (1.21, 1.07), 160
// 14.3 and 13.5 (1.14, 1.03): the line is drawn by the widest rows, and 160 and 192
// columns are on its slower side.
constexpr int kTilesFrom = 5;
constexpr int kPW = 8;      // producer warps
constexpr int kGPitch = kRound + 2;  // row stride of the pairs' dots
constexpr int kHalf = kRound / 2;
constexpr int kMPitch = kRound + 4;  // row strides of M and of the inverses: 16-byte reads of
constexpr int kWPitch = kHalf + 4;   // eight rows fall in distinct banks

// Columns per lane, warps that share out the columns, and groups of such warps:
// two groups split the dots (with q, with the q^f rows) and the bins. Odd widths
// are padded with a zero stripe in shared memory.
__host__ __device__ constexpr int lane_cols(int vpl) { return vpl == 1 ? 1 : 2; }
__host__ __device__ constexpr int group_warps(int vpl) { return (vpl + lane_cols(vpl) - 1) / lane_cols(vpl); }
__host__ __device__ constexpr int groups(int vpl) { return vpl >= 5 ? 1 : 2; }
__host__ __device__ constexpr int consumers(int vpl) { return groups(vpl) * group_warps(vpl); }
__host__ __device__ constexpr int item_threads(int vpl) { return (consumers(vpl) + kPW) * 32; }

// A round's vectors, by rating unless said otherwise.
enum {
    vBase = 0,  // gbias + bu_t - residual (with the ordinal head gbias + bu_t)
    vCu,        // cu_t
    vWq,        // -lr_i a_i^(m-1-k)
    vWf,        // -lr_iqf a_f^(later ratings of the bin)
    vBe,        // a_f^(earlier ratings of the bin)
    vOff,       // the q^f row's offset in shared memory
    vBins,      // time bin | frequency bin << 8 | slot << 16
    vSameT,     // the ratings of the same time bin
    vSameF,     // ... frequency bin
    vTarget,    // the raw rating (ordinal head)
    vUnscale,   // the inverse of the pe row's scale
    vSlotOff,   // by slot (the round's bins, in order of their first rating): the row's offset,
    vSlotDec,   // ... a_f^(ratings of the bin) - 1
    vSlots,     // [0]: the number of slots
    kVecs
};

// Columns in shared memory, and the row stride of pe and q^f rows: 16-byte reads
// of rows k and k + 1 fall in distinct halves of the banks.
__host__ __device__ constexpr uint32_t smem_cols(uint32_t Fs) { return Fs == 32 ? 32 : (Fs + 63) / 64 * 64; }
__host__ __device__ constexpr uint32_t row_pitch(uint32_t Fs) { return smem_cols(Fs) + 16; }
struct ItemSmem {  // offsets in floats, multiples of 4
    uint32_t pe, qf, q, m, w, vec, gp, pd, xs, u, bias, cx, wb, pow, total;
};
__host__ __device__ inline ItemSmem item_smem(uint32_t Fs, uint32_t NF, uint32_t cw) {
    ItemSmem L;
    const uint32_t P = row_pitch(Fs);
    uint32_t o = 0;
    L.pe = o;   o += 3 * kRound * P;                // three rounds of pe rows
    L.qf = o;   o += NF * P;                        // the item's q^f rows
    L.q = o;    o += smem_cols(Fs);                 // q at the round's start
    L.m = o;    o += 3 * kRound * kMPitch;          // three rounds of M (row j: M_ji)
    L.w = o;    o += 2 * kRound * kWPitch;          // two rounds of the diagonal blocks' inverses
    L.vec = o;  o += 5 * kVecs * kRound;            // five rounds of vectors
    L.gp = o;   o += 3 * kRound * kGPitch;          // the pairs' dots, over each third of the columns
    L.pd = o;   o += cw * kRound;                   // consumers' partial dots
    L.xs = o;   o += cw * kRound;                   // a consumer's C and errors
    L.u = o;    o += (kRound + 1) * kRound;         // update weights: q's, then by slot (zero outside the bin)
    L.bias = o; o += 132;                           // ib, bit_bin[64], ibias_freq[64]
    L.cx = o;   o += kRound;                        // C's part without the dots
    L.wb = o;   o += kRound;                        // err cu of the round before
    L.pow = o;  o += 8 * 36;                        // a_i^n, a_f^n, a_i^n - 1, a_f^n - 1, n = 0 .. kRound; rounded a
    L.total = o;
    return L;
}

// One producer's rows of a round, asked for a step ahead.
template <int VPL, int MODE>
struct Rows {
    Vec<VPL> x[4], y[4];
    Vec<MODE == kPerDay ? VPL : 1> d[MODE == kPerDay ? 4 : 1], c[MODE == kPerDay ? 4 : 1];
};

struct ItemCtx {
    const DeviceState& s;
    const EpochParams& p;
    const Bf16Copies& bf;
    float* smem;
    ItemSmem L;
    uint64_t a, n;    // the item's ratings in irec
    uint32_t rounds;
    uint32_t pitch;
    const float *apow, *fpow, *adec, *fdec;
    bool ordinal;
};

__device__ __forceinline__ int round_len(const ItemCtx& c, uint32_t r) {
    const uint64_t left = c.n - (uint64_t)r * kRound;
    return (int)(left < (uint64_t)kRound ? left : kRound);
}

// Round r's records, one per lane. Lanes past the item's end take its last
// record, so that no load of a round stands behind a branch; their weights are
// zero.
__device__ __forceinline__ Rec round_rec(const ItemCtx& c, uint32_t r, int lane) {
    const uint64_t at = (uint64_t)r * kRound + lane;
    return load_rec(c.s.irec + c.a + (at < c.n ? at : c.n - 1));
}

// The user rows of ratings pw, pw + 8, pw + 16, pw + 24.
template <int VPL, int MODE>
__device__ __forceinline__ void ask_rows(const ItemCtx& c, const Rec& rec, int pw, int lane, Rows<VPL, MODE>& R) {
    const DeviceState& s = c.s;
    const uint32_t Fs = s.Fs;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t u = rec_id(__shfl_sync(kFull, rec.key, pw + kPW * k));
        if constexpr (MODE == kBf16) {
            R.x[k].load_bf16(c.bf.pyc + (size_t)u * Fs, lane);
            R.y[k].load_bf16(c.bf.ufeat2 + (size_t)u * Fs, lane);
        } else {
            R.x[k].load_nc(s.pyc + (size_t)u * Fs, lane);
            R.y[k].load_nc(s.ufeat2 + (size_t)u * Fs, lane);
        }
        if constexpr (MODE == kPerDay) {
            const uint32_t ud = __shfl_sync(kFull, rec.ud, pw + kPW * k);
            const uint32_t at = ud < s.n_ud ? ud : 0u;
            R.d[k].load_nc(s.ufeat_day + (size_t)at * Fs, lane);
            R.c[k].load_nc(s.ycache_day + (size_t)at * Fs, lane);
        }
    }
}

// The user-side scalars of the lane's rating: bu_t's and cu_t's terms
// (src/tsvdx4p.rs:690-708).
__device__ __forceinline__ void ask_scalars(const ItemCtx& c, const Rec& r, float (&us)[7]) {
    const DeviceState& s = c.s;
    const uint32_t u = rec_id(r.key), ud = r.ud < s.n_ud ? r.ud : 0u;
    us[0] = __ldg(s.ubias + u);
    us[1] = __ldg(s.but_bin + (size_t)u * s.T + rec_tbin(r.key));
    us[2] = __ldg(s.alpha_u + u);
    us[3] = __ldg(s.ubias_day + ud);
    us[4] = __ldg(s.ycache_bias + u);
    us[5] = __ldg(s.cu + u);
    us[6] = __ldg(s.cut + ud);
}

// Producer warp pw, round r: the pe rows of its ratings; the last one also the
// round's user-side scalars.
template <int VPL, int MODE>
__device__ __forceinline__ void stage(const ItemCtx& c, uint32_t r, int pw, int lane, const Rec& rec,
                                      const float (&us)[7], Rows<VPL, MODE>& R) {
    const DeviceState& s = c.s;
    const uint32_t P = c.pitch;
    float* pe = c.smem + c.L.pe + (r % 3) * kRound * P;
    float* V = c.smem + c.L.vec + (r % 5) * kVecs * kRound;
    if (pw == kPW - 1) {
        const bool hud = rec.ud < s.n_ud;
        const float bu = us[0] + us[1] + us[2] * rec.dev + (hud ? us[3] : 0.0f) + us[4];
        V[vBase * kRound + lane] = c.ordinal ? s.gbias + bu : s.gbias + bu - rec.res;
        V[vCu * kRound + lane] = us[5] + (hud ? us[6] : 0.0f);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = pw + kPW * k;
        R.x[k].fma(__shfl_sync(kFull, rec.dev, j), R.y[k]);
        if constexpr (MODE == kPerDay) {
            const float h = __shfl_sync(kFull, rec.ud, j) < s.n_ud ? 1.0f : 0.0f;
            R.x[k].fma(h, R.d[k]);
            R.x[k].fma(h, R.c[k]);
        }
        R.x[k].store(pe + (uint32_t)j * P, lane);
        float x[VPL];
        R.x[k].to(x);
        const float unscale = row_unscale(x);
        if (lane == 0) V[vUnscale * kRound + j] = unscale;
    }
}

// Producer warps 0-5, round r: three 16 x 8 tiles of the pairs' dots over a third
// of the columns and, once all are there, some rows of M.
template <int VPL>
__device__ __forceinline__ void make_m(const ItemCtx& c, uint32_t r, int pw, int lane) {
    const EpochParams& p = c.p;
    const uint32_t P = c.pitch;
    const float* pe = c.smem + c.L.pe + (r % 3) * kRound * P;
    const float* V = c.smem + c.L.vec + (r % 5) * kVecs * kRound;
    float* G = c.smem + c.L.gp;
    {
        // Tiles of G = PE PE^T that hold every pair: rows 0-15 with columns 0-7,
        // 8-15, 16-23 (warps 0-2), rows 0-15 with 24-31, rows 16-31 with 16-23,
        // 24-31 (warps 3-5), from FP16 parts, split on the way in. A lane reads 4
        // consecutive values as the k indices (2t, 2t+1, 2t+8, 2t+9) of a 16-column
        // step, for both operands alike, so a row's fragment serves as either.
        const int third = pw % 3;
        const bool low = pw >= 3;
        const int g = lane >> 2, t = lane & 3;
        const float* row = pe + (uint32_t)g * P + 4 * t;
        float d[3][3][4] = {}, scale[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) scale[x] = row_scale(V[vUnscale * kRound + g + 8 * x]);
#pragma unroll 1
        for (int ks = third * (2 * VPL) / 3; ks < (third + 1) * (2 * VPL) / 3; ++ks) {
            // fragments of rows 0-7, 8-15, 16-23, 24-31: {lo pair, hi pair} of k
            uint32_t h[4][2], l[4][2];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (x < 3 || low) {
                    const float4 v = *reinterpret_cast<const float4*>(row + (uint32_t)(8 * x) * P + 16 * ks);
                    split_pair(v.x * scale[x], v.y * scale[x], h[x][0], l[x][0]);
                    split_pair(v.z * scale[x], v.w * scale[x], h[x][1], l[x][1]);
                }
            }
            const uint32_t ah[4] = {h[0][0], h[1][0], h[0][1], h[1][1]}, al[4] = {l[0][0], l[1][0], l[0][1], l[1][1]};
            auto tile = [&](float (&acc)[3][4], const uint32_t (&xh)[4], const uint32_t (&xl)[4], int b) {
                mma_f16(acc[0], xl, h[b][0], h[b][1]);
                mma_f16(acc[1], xh, l[b][0], l[b][1]);
                mma_f16(acc[2], xh, h[b][0], h[b][1]);
            };
            if (!low) {
                tile(d[0], ah, al, 0);
                tile(d[1], ah, al, 1);
                tile(d[2], ah, al, 2);
            } else {
                const uint32_t ch[4] = {h[2][0], h[3][0], h[2][1], h[3][1]}, cl[4] = {l[2][0], l[3][0], l[2][1], l[3][1]};
                tile(d[0], ah, al, 3);
                tile(d[1], ch, cl, 2);
                tile(d[2], ch, cl, 3);
            }
        }
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = (low && x > 0 ? 16 : 0) + g + 8 * (e >> 1);
                const int j = (low ? (x == 1 ? 16 : 24) : 8 * x) + 2 * t + (e & 1);
                G[(third * kRound + i) * kGPitch + j] = (d[x][0][e] + d[x][1][e]) + d[x][2][e];
            }
    }
    asm volatile("bar.sync 3, 192;" ::: "memory");
    // M_ji (i < j): the effect of err_i on rating j through q, the q^f row of a
    // shared bin and the item biases; lane = i, rows j = pw, pw + 6, ...
    float* M = c.smem + c.L.m + (r % 3) * kRound * kMPitch;
    const int m = round_len(c, r);
    const float cui = V[vCu * kRound + lane];
    const uint32_t bi = __float_as_uint(V[vBins * kRound + lane]);
    const unsigned after = ~((2u << lane) - 1u);
    const float* Gi = G + lane * kGPitch;
    const float unscale = V[vUnscale * kRound + lane];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int j = pw + 6 * k;
        if (k < 5 || j < kRound) {
            const uint32_t bj = __float_as_uint(V[vBins * kRound + j]);
            const unsigned same = __float_as_uint(V[vSameF * kRound + j]);
            const float g = ((Gi[j] + Gi[kRound * kGPitch + j]) + Gi[2 * kRound * kGPitch + j]) * unscale * V[vUnscale * kRound + j];
            const bool same_f = (same >> lane & 1u) != 0u, same_t = ((bi ^ bj) & 0xffu) == 0u;
            const float ai = c.apow[max(j - 1 - lane, 0)];
            const float af = c.fpow[__popc(same & after & ((1u << j) - 1u))];
            const float lr_bias = p.lr_ib + (same_t ? p.lr_ti : 0.0f) + (same_f ? p.lr_ibf : 0.0f);
            const float lr_row = p.lr_i * ai + (same_f ? p.lr_iqf * af : 0.0f);
            M[j * kMPitch + lane] = lane < j && j < m ? V[vCu * kRound + j] * cui * lr_bias + lr_row * g : 0.0f;
        }
    }
}

// Producer 7: round r's weights and bins, from its records (every vector but the
// user-side scalars).
__device__ __forceinline__ void make_vectors(const ItemCtx& c, uint32_t r, int lane, const Rec& rec) {
    float* V = c.smem + c.L.vec + (r % 5) * kVecs * kRound;
    const int m = round_len(c, r);
    const bool valid = lane < m;
    const uint32_t fb = rec_fbin(rec.key), tb = rec_tbin(rec.key);
    const unsigned same = __match_any_sync(kFull, valid ? fb : 64u + (uint32_t)lane);
    const unsigned same_t = __match_any_sync(kFull, valid ? tb : 64u + (uint32_t)lane);
    const unsigned below = (1u << lane) - 1u;
    const int earlier = __popc(same & below), in_bin = __popc(same);
    // slots: the bins in order of their first rating
    const unsigned firsts = __ballot_sync(kFull, valid && earlier == 0);
    const int slot = __popc(firsts & ((1u << (__ffs((int)same) - 1)) - 1u));
    const uint32_t off = valid ? fb * c.pitch : 0u;
    V[vWq * kRound + lane] = valid ? -c.p.lr_i * c.apow[m - 1 - lane] : 0.0f;
    V[vWf * kRound + lane] = valid ? -c.p.lr_iqf * c.fpow[in_bin - 1 - earlier] : 0.0f;
    V[vBe * kRound + lane] = c.fpow[earlier];
    V[vOff * kRound + lane] = __uint_as_float(off);
    V[vBins * kRound + lane] = __uint_as_float(tb | fb << 8 | (uint32_t)(valid ? slot : 32) << 16);
    V[vSameT * kRound + lane] = __uint_as_float(same_t);
    V[vSameF * kRound + lane] = __uint_as_float(same);
    V[vTarget * kRound + lane] = rec.res;
    if (valid && earlier == 0) {
        V[vSlotOff * kRound + slot] = __uint_as_float(off);
        V[vSlotDec * kRound + slot] = c.fdec[in_bin];
    }
    if (lane == 0) V[vSlots * kRound] = __int_as_float(__popc(firsts));
}

// The item's biases after the round whose vectors are V and whose err cu are in
// wb (ratings of one bin write the same value).
__device__ __forceinline__ void bias_update(const ItemCtx& c, const float* V, int m, int lane) {
    float* bias = c.smem + c.L.bias;
    const float4* wb = reinterpret_cast<const float4*>(c.smem + c.L.wb);
    const unsigned st = __float_as_uint(V[vSameT * kRound + lane]), sf = __float_as_uint(V[vSameF * kRound + lane]);
    const uint32_t bins = __float_as_uint(V[vBins * kRound + lane]);
    const uint32_t tb = bins & 0xffu, fb = bins >> 8 & 0xffu;
    float all = 0.0f, t = 0.0f, f = 0.0f;
#pragma unroll 4
    for (int q = 0; q < kRound / 4; ++q) {
        const float4 w4 = wb[q];
        const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = 4 * q + e;
            all += w[e];
            t += (st >> k & 1u) ? w[e] : 0.0f;
            f += (sf >> k & 1u) ? w[e] : 0.0f;
        }
    }
    const float nt = bias[1 + tb] - c.p.lr_ti * t, nf = bias[65 + fb] - c.p.lr_ibf * f;
    __syncwarp();
    if (lane < m) {
        bias[1 + tb] = nt;
        bias[65 + fb] = nf;
    }
    if (lane == 0) bias[0] -= c.p.lr_ib * all;
    __syncwarp();
}

// The inverses of I + M's two diagonal 16 x 16 blocks of round r: lane = column,
// forward substitution over the block's rows.
__device__ __forceinline__ void invert_blocks(const ItemCtx& c, uint32_t r, int lane) {
    const int b0 = lane & kHalf, col = lane & (kHalf - 1);
    const float* M = c.smem + c.L.m + (r % 3) * kRound * kMPitch + b0 * kMPitch + b0;
    float* W = c.smem + c.L.w + (r & 1) * kRound * kWPitch + b0 * kWPitch + col;
    float w[kHalf];
#pragma unroll
    for (int j = 0; j < kHalf; ++j) {
        float a0 = j == col ? 1.0f : 0.0f, a1 = 0.0f;
#pragma unroll
        for (int q = 0; 4 * q < j; ++q) {
            const float4 m4 = *reinterpret_cast<const float4*>(M + j * kMPitch + 4 * q);
            a0 = fmaf(-m4.x, w[4 * q], a0);
            if (4 * q + 1 < j) a1 = fmaf(-m4.y, w[4 * q + 1], a1);
            if (4 * q + 2 < j) a0 = fmaf(-m4.z, w[4 * q + 2], a0);
            if (4 * q + 3 < j) a1 = fmaf(-m4.w, w[4 * q + 3], a1);
        }
        w[j] = a0 + a1;
    }
#pragma unroll
    for (int j = 0; j < kHalf; ++j) W[j * kWPitch] = w[j];
}

// Sixteen products with sixteen consecutive floats of shared memory.
__device__ __forceinline__ float dot16(const float (&w)[kHalf], const float* x) {
    float e0 = 0.0f, e1 = 0.0f, e2 = 0.0f, e3 = 0.0f;
#pragma unroll
    for (int k = 0; k < kHalf; k += 4) {
        const float4 b = *reinterpret_cast<const float4*>(x + k);
        e0 = fmaf(w[k], b.x, e0);
        e1 = fmaf(w[k + 1], b.y, e1);
        e2 = fmaf(w[k + 2], b.z, e2);
        e3 = fmaf(w[k + 3], b.w, e3);
    }
    return (e0 + e1) + (e2 + e3);
}

// Consumer warp cw, round r, with columns from col0 on. WQ: the warp takes the
// dots with q and its update; WF: those with the q^f rows; the slots slot0, slot0
// + slot_step, ... are its to update. qv: the lane's columns of q.
template <int VPL, bool WQ, bool WF>
__device__ __forceinline__ void consume(const ItemCtx& c, uint32_t r, int cw, int lane, int col0, int slot0,
                                        float (&qv)[lane_cols(VPL)], const float (&th)[4]) {
    constexpr int CW = consumers(VPL), CPL = lane_cols(VPL), KS = 2 * CPL;  // 16-column steps of the warp's columns
    constexpr int NG = groups(VPL);
    const uint32_t P = c.pitch;
    const float* pe = c.smem + c.L.pe + (r % 3) * kRound * P;
    const float* V = c.smem + c.L.vec + (r % 5) * kVecs * kRound;
    const float* M = c.smem + c.L.m + (r % 3) * kRound * kMPitch;
    const float* W = c.smem + c.L.w + (r & 1) * kRound * kWPitch;
    float* qf = c.smem + c.L.qf;
    float* q = c.smem + c.L.q;
    float* xs = c.smem + c.L.xs + cw * kRound;
    float* U = c.smem + c.L.u;
    const int m = round_len(c, r);
    // partial dots of the warp's columns: lane (g, t) takes columns 4t..4t+3 of
    // each step for ratings g, g + 8, g + 16, g + 24
    {
        const int g = lane >> 2, t = lane & 3;
        f32x2 s1[4], s2[4];
        const float* row[4];
        const float* er = pe + (uint32_t)g * P + col0 + 4 * t;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            s1[x] = s2[x] = 0ull;
            if constexpr (WF) row[x] = qf + __float_as_uint(V[vOff * kRound + g + 8 * x]) + col0 + 4 * t;
        }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            ulonglong2 f;
            if constexpr (WQ) f = *reinterpret_cast<const ulonglong2*>(q + col0 + 4 * t + 16 * ks);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(er + (uint32_t)(8 * x) * P + 16 * ks);
                if constexpr (WQ) {
                    s1[x] = fma2(e.x, f.x, s1[x]);
                    s1[x] = fma2(e.y, f.y, s1[x]);
                }
                if constexpr (WF) {
                    const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(row[x] + 16 * ks);
                    s2[x] = fma2(e.x, h.x, s2[x]);
                    s2[x] = fma2(e.y, h.y, s2[x]);
                }
            }
        }
        float v[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            float a, b;
            v[x] = 0.0f;
            if constexpr (WQ) {
                unpack2(s1[x], a, b);
                v[x] = c.apow[g + 8 * x] * (a + b);
            }
            if constexpr (WF) {
                unpack2(s2[x], a, b);
                v[x] = fmaf(V[vBe * kRound + g + 8 * x], a + b, v[x]);
            }
        }
        // sums over t; lane (g, t) ends with rating g + 8 t
#pragma unroll
        for (int o = 2; o > 0; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < o; ++k) {
                const float keep = up ? v[k + o] : v[k], send = up ? v[k] : v[k + o];
                v[k] = keep + __shfl_xor_sync(kFull, send, o);
            }
        }
        c.smem[c.L.pd + cw * kRound + g + 8 * t] = v[0];
    }
    // ahead of their use: the lane's row of its diagonal block's inverse and of the
    // block below the first, the round's values of the lane's columns
    float wd[kHalf], wm[kHalf];
#pragma unroll
    for (int k = 0; k < kHalf; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(W + lane * kWPitch + k);
        wd[k] = a.x; wd[k + 1] = a.y; wd[k + 2] = a.z; wd[k + 3] = a.w;
        const float4 b = *reinterpret_cast<const float4*>(M + lane * kMPitch + k);
        wm[k] = b.x; wm[k + 1] = b.y; wm[k + 2] = b.z; wm[k + 3] = b.w;
    }
    const int col = col0 + CPL * lane;
    float e[kRound][CPL];
#pragma unroll
    for (int k = 0; k < kRound; ++k) {
        const float* pc = pe + (uint32_t)k * P + col;
        if constexpr (CPL == 2) {
            const float2 t = *reinterpret_cast<const float2*>(pc);
            e[k][0] = t.x;
            e[k][CPL - 1] = t.y;
        } else {
            e[k][0] = *pc;
        }
    }
    const float wq = V[vWq * kRound + lane], wf = V[vWf * kRound + lane], cu = V[vCu * kRound + lane];
    const int slot = (int)(__float_as_uint(V[vBins * kRound + lane]) >> 16);
    const int slots = __float_as_int(V[vSlots * kRound]);
    const bool valid = lane < m;
    // all partial dots, and producer 6's part of C, are in place
    asm volatile("bar.sync 1, %0;" ::"n"((CW + 1) * 32) : "memory");
    float x = c.smem[c.L.cx + lane];
    {
        float dot = 0.0f;
#pragma unroll
        for (int w = 0; w < CW; ++w) dot += c.smem[c.L.pd + w * kRound + lane];
        x += dot;
    }
    float err = 0.0f;
    if (!c.ordinal) {
        // the first block's errors, their effect on the second block, its errors
        xs[lane] = x = valid ? x : 0.0f;
        __syncwarp();
        err = dot16(wd, xs);
        __syncwarp();
        if (lane < kHalf) xs[lane] = err;
        __syncwarp();
        x -= dot16(wm, xs);
        if (lane >= kHalf) xs[lane] = x;
        __syncwarp();
        const float e1 = dot16(wd, xs + kHalf);
        if (lane >= kHalf) err = e1;
    } else {
        const int y = (int)V[vTarget * kRound + lane];
        // four steps in straight-line code, their entries of M asked for at once (3 M
        // ratings, f = 20: 6.0 ms against 6.4 one by one)
#pragma unroll 1
        for (int k0 = 0; k0 < kRound; k0 += 4) {
            const float4 m4 = *reinterpret_cast<const float4*>(M + lane * kMPitch + k0);
            const float mk[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float ek = valid ? ordinal_grad(th, x, y) : 0.0f;
                if (k0 + e == lane) err = ek;
                x = fmaf(k0 + e < lane ? -mk[e] : 0.0f, __shfl_sync(kFull, ek, k0 + e), x);
            }
        }
    }
    // the updates' weights, every warp some rows of the table
    for (int k = cw; k <= slots; k += CW)
        U[k * kRound + lane] = k == 0 ? wq * err : slot == k - 1 ? wf * err : 0.0f;
    if (cw == CW - 1) c.smem[c.L.wb + lane] = valid ? err * cu : 0.0f;
    if constexpr (CW > 1) asm volatile("bar.sync 4, %0;" ::"n"(CW * 32) : "memory");
    else __syncwarp();
    // sums of the lane's columns weighted by a row of the table
    auto weighted = [&](const float* w, float (&a)[CPL]) {
        float b[4][CPL];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < CPL; ++v) b[u][v] = 0.0f;
#pragma unroll
        for (int k = 0; k < kRound; k += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
            for (int v = 0; v < CPL; ++v) {
                b[0][v] = fmaf(w4.x, e[k][v], b[0][v]);
                b[1][v] = fmaf(w4.y, e[k + 1][v], b[1][v]);
                b[2][v] = fmaf(w4.z, e[k + 2][v], b[2][v]);
                b[3][v] = fmaf(w4.w, e[k + 3][v], b[3][v]);
            }
        }
#pragma unroll
        for (int v = 0; v < CPL; ++v) a[v] = (b[0][v] + b[1][v]) + (b[2][v] + b[3][v]);
    };
    // a row's change, its decay (a^n - 1) x among it, is rounded into the row once
    if constexpr (WQ) {
        float a[CPL];
        weighted(U, a);
        const float d = c.adec[m];
#pragma unroll
        for (int v = 0; v < CPL; ++v) q[col + v] = qv[v] = qv[v] + fmaf(d, qv[v], a[v]);
    }
#pragma unroll 1
    for (int k = slot0; k < slots; k += NG) {
        float a[CPL];
        weighted(U + (k + 1) * kRound, a);
        float* row = qf + __float_as_uint(V[vSlotOff * kRound + k]) + col;
        const float d = V[vSlotDec * kRound + k];
#pragma unroll
        for (int v = 0; v < CPL; ++v) {
            const float o = row[v];
            row[v] = o + fmaf(d, o, a[v]);
        }
    }
    __syncwarp();
}

template <int VPL, int MODE>
__global__ void __launch_bounds__(item_threads(VPL), 1) k_item_rounds(DeviceState s, EpochParams p,
                                                                                   Bf16Copies bf) {
    extern __shared__ __align__(16) float smem[];
    __shared__ uint32_t sh_next[2];
    constexpr int CW = consumers(VPL), GW = group_warps(VPL), CPL = lane_cols(VPL);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t Fs = s.Fs, NF = s.NF, T = s.T;
    ItemCtx c{s, p, bf, smem, item_smem(Fs, NF, CW), 0, 0, 0, row_pitch(Fs), nullptr, nullptr, nullptr, nullptr, s.raw != nullptr};
    if (threadIdx.x == 64) sh_next[1] = atomicAdd(&s.counters[2], 1u);
    if (threadIdx.x < 2) decay_powers<kRound>(smem + c.L.pow + threadIdx.x * 144, p, threadIdx.x == 1);
    // the zero columns of an odd width (those of q and q^f come with each item: an
    // update by a weight that is not finite leaves them not zero)
    if constexpr (VPL > 1 && (VPL & 1)) {
        const uint32_t P = row_pitch(Fs);
        for (uint32_t e = threadIdx.x; e < 3 * kRound * 32; e += blockDim.x) smem[c.L.pe + e / 32 * P + Fs + e % 32] = 0.0f;
    }
    float th[4];
    load_thresholds(s, th);
    __syncthreads();
    const int pw = warp - CW;
    float* bias = smem + c.L.bias;
    // Items heaviest first, each to the next block that is free. Where several passes
    // share the GPU (tsvd_group.cu) not every block of a pass is there from the start,
    // and one that owned an item would keep it waiting (eight variants of 1 M ratings,
    // up to 128 columns: 6.9 ms an epoch with the first items bound to blocks, 6.4 so).
    uint32_t k = sh_next[1];
    // light items one warp each; with the per-day rows every item goes in rounds
    const uint32_t heavy_min = MODE == kPerDay ? 1u : max(s.heavy_min, 1u);
    for (uint32_t turn = 0; k < s.n_item_work; ++turn) {
        const uint32_t i = s.item_work[k];
        c.a = s.item_off[i];
        c.n = s.item_off[i + 1] - c.a;
        if (c.n < heavy_min) break;  // heaviest first
        c.apow = smem + c.L.pow + (c.n >= s.rounded_decay_min ? 144 : 0);
        c.fpow = c.apow + 36;
        c.adec = c.apow + 72;
        c.fdec = c.apow + 108;
        c.rounds = (uint32_t)((c.n + kRound - 1) / kRound);
        const int last = (int)c.rounds - 1;
        if (warp < CW) {
            // consumers: their columns of the item's q and q^f rows
            constexpr bool two = groups(VPL) == 2;
            const int col0 = (warp % GW) * 32 * CPL, col = col0 + CPL * lane;
            const bool here = (uint32_t)col < Fs, first = warp < GW;  // the first group: q and its dots
            float qv[CPL];
#pragma unroll
            for (int v = 0; v < CPL; ++v) qv[v] = 0.0f;
            if (first) {
#pragma unroll
                for (int v = 0; v < CPL; ++v)
                    smem[c.L.q + col + v] = qv[v] = here ? __ldcg(s.ifeat + (size_t)i * Fs + col + v) : 0.0f;
            }
            if (!two || !first) {
#pragma unroll 4
                for (uint32_t b = 0; b < NF; ++b)
#pragma unroll
                    for (int v = 0; v < CPL; ++v)
                        smem[c.L.qf + b * c.pitch + col + v] =
                            here ? __ldcg(s.ifeat_freq + ((size_t)i * NF + b) * Fs + col + v) : 0.0f;
            }
            __syncwarp();
            __syncthreads();
            __syncthreads();
            for (int t = 0; t <= last; ++t) {
                if constexpr (two) {
                    if (first) consume<VPL, true, false>(c, (uint32_t)t, warp, lane, col0, 1, qv, th);
                    else consume<VPL, false, true>(c, (uint32_t)t, warp, lane, col0, 0, qv, th);
                } else {
                    consume<VPL, true, true>(c, (uint32_t)t, warp, lane, col0, 0, qv, th);
                }
                __syncthreads();
            }
            if (here && first) {
#pragma unroll
                for (int v = 0; v < CPL; ++v) s.ifeat[(size_t)i * Fs + col + v] = qv[v];
            }
            if (here && (!two || !first)) {
#pragma unroll 4
                for (uint32_t b = 0; b < NF; ++b)
#pragma unroll
                    for (int v = 0; v < CPL; ++v)
                        __stcg(s.ifeat_freq + ((size_t)i * NF + b) * Fs + col + v, smem[c.L.qf + b * c.pitch + col + v]);
            }
            __syncwarp();
        } else {
            Rec rec = round_rec(c, 0, lane), ahead = round_rec(c, 1, lane);
            float us[7] = {};
            Rows<VPL, MODE> R;
            if (pw == kPW - 1) ask_scalars(c, rec, us);
            ask_rows<VPL, MODE>(c, rec, pw, lane, R);
            if (pw == 7) make_vectors(c, 0, lane, rec);
            if (pw == 6) {
                if (lane == 0) {
                    sh_next[turn & 1] = atomicAdd(&s.counters[2], 1u);
                    bias[0] = __ldcg(s.ibias + i);
                }
                for (uint32_t e = lane; e < 64; e += 32) {
                    bias[1 + e] = e < T ? __ldcg(s.bit_bin + (size_t)i * T + e) : 0.0f;
                    bias[65 + e] = e < NF ? __ldcg(s.ibias_freq + (size_t)i * NF + e) : 0.0f;
                }
                __syncwarp();
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kPW * 32) : "memory");
            // The next round's rows: asked for before the pairs' dots where they are
            // long (1 KB rows that miss L2 need the time), after them where the
            // registers they would hold cost more (f <= 128).
            constexpr bool kAskEarly = VPL >= 5;
            auto ask_next = [&] {
                if (pw == kPW - 1) ask_scalars(c, rec, us);
                ask_rows<VPL, MODE>(c, rec, pw, lane, R);
            };
            for (int t = -2; t <= last; ++t) {
                const uint32_t r = (uint32_t)(t + 2);
                const bool more = r < c.rounds;
                if (more) {
                    stage<VPL, MODE>(c, r, pw, lane, rec, us, R);
                    rec = ahead;
                    if constexpr (kAskEarly) ask_next();
                    ahead = round_rec(c, r + 2, lane);
                    asm volatile("bar.sync 2, %0;" ::"n"(kPW * 32) : "memory");
                }
                if (pw < 6) {
                    if (more) make_m<VPL>(c, r, pw, lane);
                } else if (pw == 6) {
                    if (t >= 0) {
                        if (t > 0)
                            bias_update(c, smem + c.L.vec + ((uint32_t)(t - 1) % 5) * kVecs * kRound, kRound, lane);
                        const float* V = smem + c.L.vec + ((uint32_t)t % 5) * kVecs * kRound;
                        const uint32_t bins = __float_as_uint(V[vBins * kRound + lane]);
                        const float bi = bias[0] + bias[1 + (bins & 0xffu)] + bias[65 + (bins >> 8 & 0xffu)];
                        smem[c.L.cx + lane] = V[vBase * kRound + lane] + bi * V[vCu * kRound + lane];
                        __syncwarp();
                        asm volatile("bar.arrive 1, %0;" ::"n"((CW + 1) * 32) : "memory");
                    }
                } else {
                    if (t + 1 >= 0 && t + 1 <= last && !c.ordinal) invert_blocks(c, (uint32_t)(t + 1), lane);
                    if (r + 1 < c.rounds) make_vectors(c, r + 1, lane, rec);
                }
                if (more && !kAskEarly) ask_next();
                __syncthreads();
            }
            if (pw == 6) {
                bias_update(c, smem + c.L.vec + ((uint32_t)last % 5) * kVecs * kRound, round_len(c, (uint32_t)last),
                            lane);
                for (uint32_t e = lane; e < 64; e += 32) {
                    if (e < T) s.bit_bin[(size_t)i * T + e] = bias[1 + e];
                    if (e < NF) s.ibias_freq[(size_t)i * NF + e] = bias[65 + e];
                }
                if (lane == 0) s.ibias[i] = bias[0];
                __syncwarp();
            }
        }
        k = sh_next[turn & 1];
        __syncthreads();  // the next item's rounds reuse the last one's vectors
    }
    if constexpr (MODE != kPerDay) {
        if (warp > 0) {
            if (lane == 0) k = atomicAdd(&s.counters[2], 1u);
            k = __shfl_sync(kFull, k, 0);
        }
        light_items<VPL, MODE == kBf16>(s, p, bf, k, lane, smem + warp * kLightRows * 2 * Fs);
    }
}

template <int VPL, int MODE>
void launch_item(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    auto kern = k_item_rounds<VPL, MODE>;
    const size_t smem = std::max<size_t>(item_smem(s.Fs, s.NF, consumers(VPL)).total,
                                         light_smem(item_threads(VPL) / 32, s.Fs)) * sizeof(float);
    allow_dyn_smem(kern, smem);
    int dev = 0, sms = 0;
    TSVD_CUDA(cudaGetDevice(&dev));
    TSVD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    kern<<<(unsigned)sms, item_threads(VPL), smem, m->stream>>>(s, p, bf);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

}  // namespace

void launch_item_stratum(tsvd_model* m, const DeviceState& s, const EpochParams& p, const Bf16Copies& bf) {
    const int vpl = (int)(s.Fs / 32);
    if (vpl >= kTilesFrom && !s.dyd_fix && !s.raw) {
        launch_item_tiles(m, s, p, bf);
    } else if (s.dyd_fix) {
        TSVD_DISPATCH(vpl, (launch_item<V, kPerDay>(m, s, p, bf)));
    } else if (bf.pyc) {
        TSVD_DISPATCH(vpl, (launch_item<V, kBf16>(m, s, p, bf)));
    } else {
        TSVD_DISPATCH(vpl, (launch_item<V, kPlain>(m, s, p, bf)));
    }
}

}  // namespace tsvd
