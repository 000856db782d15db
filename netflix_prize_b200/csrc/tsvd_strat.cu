// Deterministic stratified schedule: the reference's own parallel epoch,
// Tsvdx4pModel::fit_epoch (src/tsvdx4p.rs:390-805):
//   user stratum  (fit_epoch_user, :390-639)  users in parallel, item tables
//                 frozen, per-user NSVD1 gradients kept for the delta sums;
//   delta apply   (apply_nsvd_deltas, :341-385) per-item sums over the item's
//                 users in by-item order, split into fixed chunks;
//   ycache rebuild (:267-300);
//   item stratum  (fit_epoch_item, :644-762)  items in parallel, user tables
//                 frozen.
// No two work units touch the same parameter and every sum has a fixed
// order, so a run is bitwise reproducible.
//
// Precision form: the frozen tables a stratum only reads are rounded to BF16
// (y_j, gathered as BF16; q_i and q^f_{i,0}, whose sum is read as FP32;
// optionally p_u + ycache_u and p2_u in the item stratum, gathered as BF16)
// and accumulated in FP32; masters stay FP32 and are the only tables written.
#include <algorithm>
#include <functional>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "rand_stream.hpp"
#include "tsvd_item.cuh"

namespace tsvd {
namespace {

// ---------------------------------------------------------------------------
// FP32 -> BF16 read copies (round to nearest even). `src_stride` lets the
// frequency-bin-0 rows of ifeat_freq ([I*NF, Fs]) be copied as an [I, Fs] table.
// ---------------------------------------------------------------------------
__global__ void k_to_bf16(const float* __restrict__ src, uint64_t rows, uint32_t Fs, uint64_t src_stride,
                          __nv_bfloat16* __restrict__ dst) {
    const uint64_t n = rows * Fs;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = e / Fs, c = e - r * Fs;
        dst[e] = __float2bfloat16_rn(src[r * src_stride + c]);
    }
}

// qe0 = q_i + q^f_{i,0}: with low_memory the user stratum trains frequency bin
// 0 only (src/tsvdx4p.rs:504-531) and reads the two rows only as this sum.
// In the precision form both addends are rounded to BF16 first.
__global__ void k_make_qe0(const float* __restrict__ ifeat, const float* __restrict__ ifeat_freq, uint64_t rows,
                           uint32_t Fs, uint32_t NF, bool bf16, float* __restrict__ qe0) {
    const uint64_t n = rows * Fs;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = e / Fs, c = e - r * Fs;
        const float q = ifeat[e], f = ifeat_freq[r * NF * Fs + c];
        qe0[e] = bf16 ? __bfloat162float(__float2bfloat16_rn(q)) + __bfloat162float(__float2bfloat16_rn(f)) : q + f;
    }
}

void make_qe0(tsvd_model* m, bool bf16);

// ---------------------------------------------------------------------------
// NSVD1 delta sums per item in two fixed-order levels: fixed chunks of
// kChunkUsers consecutive by-item entries are summed by one warp each
// (k_y_partial), then each item adds its chunk partials in chunk order and
// applies the update (k_y_combine).
// ---------------------------------------------------------------------------
// Entries whose user lies outside [u_lo, u_hi) are left out (a user block; the
// full range otherwise). An item's entries are sorted by user, so the ones
// kept are contiguous and keep their order. With `accumulate` the block's
// partial is added to the chunk's earlier blocks' (blocks in user order), and
// chunks without entries in the block are left alone: passes over user blocks
// whose g_user rows fit in L2 gather from L2 instead of HBM.
template <int VPL>
// split (optional): per chunk, the first entry of each pass's user block
// (split[c * (passes + 1) + k]); without it the block's range is searched.
__global__ void __launch_bounds__(kThreads) k_y_partial(DeviceState s, uint32_t u_lo, uint32_t u_hi,
                                                        int accumulate, const uint64_t* __restrict__ split,
                                                        uint32_t passes, uint32_t pass) {
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs;
    constexpr int B = 8;  // rows in flight per warp
    for (;;) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(&s.counters[1], 1u);
        c = __shfl_sync(kFull, c, 0);
        if (c >= s.n_chunks) break;
        uint64_t a = s.chunk_lo[c];
        uint64_t b = s.chunk_lo[c + 1];
        if (b - a > kChunkUsers) b = a + kChunkUsers;
        if (split) {
            a = split[(size_t)c * (passes + 1) + pass];
            b = split[(size_t)c * (passes + 1) + pass + 1];
            if (accumulate && a == b) continue;
        } else if (u_lo != 0 || u_hi != 0xffffffffu) {
            // the chunk's entries of users u_lo..u_hi-1 (sorted by user)
            uint64_t lo = a, hi = b;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (rec_id(__ldg(&s.irec[mid].key)) < u_lo) lo = mid + 1;
                else hi = mid;
            }
            uint64_t lo2 = lo, hi2 = b;
            while (lo2 < hi2) {
                const uint64_t mid = (lo2 + hi2) >> 1;
                if (rec_id(__ldg(&s.irec[mid].key)) < u_hi) lo2 = mid + 1;
                else hi2 = mid;
            }
            a = lo;
            b = lo2;
            if (accumulate && a == b) continue;
        }
        // rows wider than 32 * VPL columns (n_feat > 256) in slices
        for (uint32_t c0 = 0; c0 < Fs; c0 += 32 * VPL) {
            float acc[VPL];
#pragma unroll
            for (int v = 0; v < VPL; ++v) acc[v] = 0.0f;
            float eacc = 0.0f;
            for (uint64_t base = a; base < b; base += 32) {
                const uint32_t cnt = (uint32_t)(b - base < 32 ? b - base : 32);
                const uint32_t mine = lane < (int)cnt ? rec_id(__ldg(&s.irec[base + lane].key)) : 0u;
                for (uint32_t j = 0; j < cnt; j += B) {
                    float g[B][VPL], e[B];
#pragma unroll
                    for (int q = 0; q < B; ++q) {
                        const uint32_t u = __shfl_sync(kFull, mine, j + q < cnt ? j + q : cnt - 1);
                        Row<VPL>::load_nc(s.g_user + (size_t)u * Fs + c0, lane, g[q]);
                        e[q] = c0 == 0 ? __ldg(s.e_user + u) : 0.0f;
                    }
#pragma unroll
                    for (int q = 0; q < B; ++q) {
                        if (j + q < cnt) {
#pragma unroll
                            for (int v = 0; v < VPL; ++v) acc[v] += g[q][v];
                            eacc += e[q];
                        }
                    }
                }
            }
            if (accumulate) {
                float prev[VPL];
                Row<VPL>::load_cg(s.chunk_part + (size_t)c * Fs + c0, lane, prev);
#pragma unroll
                for (int v = 0; v < VPL; ++v) acc[v] = prev[v] + acc[v];
                if (c0 == 0) eacc = __ldcg(s.chunk_epart + c) + eacc;
            }
            Row<VPL>::store(s.chunk_part + (size_t)c * Fs + c0, lane, acc);
            if (lane == 0 && c0 == 0) s.chunk_epart[c] = eacc;
        }
    }
}

// split[c * (nb) + k] = the first entry of chunk c whose user is >= bounds[k]
// (the chunk's entries are sorted by user).
__global__ void k_chunk_splits(DeviceState s, const uint32_t* __restrict__ bounds, uint32_t nb,
                               uint64_t* __restrict__ split) {
    const uint64_t n = (uint64_t)s.n_chunks * nb;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)(e / nb), k = (uint32_t)(e % nb);
        uint64_t lo = s.chunk_lo[c], hi = s.chunk_lo[c + 1];
        if (hi - lo > kChunkUsers) hi = lo + kChunkUsers;
        const uint32_t u = bounds[k];
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (rec_id(__ldg(&s.irec[mid].key)) < u) lo = mid + 1;
            else hi = mid;
        }
        split[e] = lo;
    }
}

// The per-chunk split table for the user-block bounds `bounds`, made when the
// bounds change (outside a stream capture; inside one, a stale table gives
// null and the passes search instead).
const uint64_t* chunk_splits(tsvd_model* m, const DeviceState& s, const std::vector<uint32_t>& bounds) {
    if (bounds != m->h_split_bounds || !m->m_chunk_split.p) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        TSVD_CUDA(cudaStreamIsCapturing(m->stream, &cs));
        if (cs != cudaStreamCaptureStatusNone) return nullptr;
        const size_t n = (size_t)s.n_chunks * bounds.size();
        if (m->m_chunk_split.bytes < n * 8) m->m_chunk_split.alloc(n * 8);
        if (m->m_split_bounds.bytes < bounds.size() * 4) m->m_split_bounds.alloc(bounds.size() * 4);
        TSVD_CUDA(cudaMemcpyAsync(m->m_split_bounds.p, bounds.data(), bounds.size() * 4, cudaMemcpyHostToDevice,
                                  m->stream));
        const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 16);
        k_chunk_splits<<<grid, 256, 0, m->stream>>>(s, m->m_split_bounds.as<uint32_t>(), (uint32_t)bounds.size(),
                                                    m->m_chunk_split.as<uint64_t>());
        TSVD_CUDA(cudaGetLastError());
        TSVD_CUDA(cudaStreamSynchronize(m->stream));  // `bounds` is the caller's
        m->launches++;
        m->h_split_bounds = bounds;
    }
    return m->m_chunk_split.as<uint64_t>();
}

// The NSVD1 delta sums of users u_lo..u_hi-1 into the chunk partials, in
// passes over user blocks of at most ~64 MB of g_user rows (L2 holds one).
// Each chunk's entries of a block come from a split table made once for the
// blocks' bounds, not from a search in every pass.
template <int VPL>
void y_partial_passes(tsvd_model* m, const DeviceState& s, uint32_t u_lo, uint32_t u_hi) {
    const uint64_t row_bytes = (uint64_t)s.Fs * 4;
    const uint32_t per = (uint32_t)std::max<uint64_t>(1, (64ull << 20) / row_bytes);
    const unsigned g = persistent_grid(k_y_partial<VPL>, 0);
    const bool whole = u_lo == 0 && u_hi >= s.n_users;
    std::vector<uint32_t> bounds;
    for (uint64_t b0 = u_lo; b0 < u_hi || b0 == u_lo; b0 += per) {
        bounds.push_back((uint32_t)b0);
        if (std::min<uint64_t>(u_hi, b0 + per) >= u_hi) break;
    }
    bounds.push_back(u_hi);
    const uint32_t passes = (uint32_t)bounds.size() - 1;
    const bool one = whole && passes == 1;  // a single pass over every user
    const uint64_t* split = one ? nullptr : chunk_splits(m, s, bounds);
    for (uint32_t k = 0; k < passes; ++k) {
        TSVD_CUDA(cudaMemsetAsync(s.counters + 1, 0, 4, m->stream));
        k_y_partial<VPL><<<g, kThreads, 0, m->stream>>>(s, one ? 0u : bounds[k], one ? 0xffffffffu : bounds[k + 1],
                                                        k == 0 ? 0 : 1, split, passes, k);
        TSVD_CUDA(cudaGetLastError());
        m->launches++;
    }
}

template <int VPL>
__global__ void __launch_bounds__(kThreads) k_y_combine(DeviceState s, EpochParams p) {
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs;
    const uint32_t warps = gridDim.x * kWarps;
    for (uint32_t i = blockIdx.x * kWarps + (threadIdx.x >> 5); i < s.n_items; i += warps) {
        const uint32_t c0 = s.item_chunk0[i], c1 = s.item_chunk0[i + 1];
        if (c0 == c1) continue;
        const float nc = (float)(s.item_off[i + 1] - s.item_off[i]);
        const float scale = p.nsvd_norm_exp == 0.0f ? 1.0f : powf(nc, p.nsvd_norm_exp);
        for (uint32_t x0 = 0; x0 < Fs; x0 += 32 * VPL) {
            float acc[VPL];
#pragma unroll
            for (int v = 0; v < VPL; ++v) acc[v] = 0.0f;
            for (uint32_t c = c0; c < c1; ++c) {
                float g[VPL];
                Row<VPL>::load_cg(s.chunk_part + (size_t)c * Fs + x0, lane, g);
#pragma unroll
                for (int v = 0; v < VPL; ++v) acc[v] += g[v];
            }
            float y[VPL];
            Row<VPL>::load_cg(s.yfeat + (size_t)i * Fs + x0, lane, y);
#pragma unroll
            for (int v = 0; v < VPL; ++v) y[v] = y[v] - p.lr_y * (acc[v] / scale + p.reg_y * y[v]);
            Row<VPL>::store(s.yfeat + (size_t)i * Fs + x0, lane, y);
            if (s.dyd_fix) {
                // per-day NSVD1 deltas, same divisor (src/tsvdx4p.rs:370-384)
                float yd[VPL];
                Row<VPL>::load_cg(s.yfeat_day + (size_t)i * Fs + x0, lane, yd);
                const unsigned long long* drow = s.dyd_fix + (size_t)i * Fs + x0;
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    const float d = (float)((double)(long long)__ldcg(drow + Row<VPL>::elem(lane, v)) / kDydScale);
                    yd[v] = yd[v] - p.lr_yd * (d / scale + p.reg_yd * yd[v]);
                }
                Row<VPL>::store(s.yfeat_day + (size_t)i * Fs + x0, lane, yd);
            }
        }
        float eacc = 0.0f;
        for (uint32_t c = c0; c < c1; ++c) eacc += __ldcg(s.chunk_epart + c);
        if (lane == 0) s.ybias[i] = s.ybias[i] - p.lr_yb * (eacc / scale);
    }
}

// A user block's NSVD1 delta sums per item (chunk partials added in chunk
// order) into sums [I, Fs] and sums_e [I], instead of applying them: the
// ranks of a sharded run add their blocks' sums before the apply.
template <int VPL>
__global__ void __launch_bounds__(kThreads) k_y_block_sums(DeviceState s, float* __restrict__ sums,
                                                           float* __restrict__ sums_e) {
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs;
    const uint32_t warps = gridDim.x * kWarps;
    for (uint32_t i = blockIdx.x * kWarps + (threadIdx.x >> 5); i < s.n_items; i += warps) {
        const uint32_t c0 = s.item_chunk0[i], c1 = s.item_chunk0[i + 1];
        for (uint32_t x0 = 0; x0 < Fs; x0 += 32 * VPL) {
            float acc[VPL];
#pragma unroll
            for (int v = 0; v < VPL; ++v) acc[v] = 0.0f;
            for (uint32_t c = c0; c < c1; ++c) {
                float g[VPL];
                Row<VPL>::load_cg(s.chunk_part + (size_t)c * Fs + x0, lane, g);
#pragma unroll
                for (int v = 0; v < VPL; ++v) acc[v] += g[v];
            }
            Row<VPL>::store(sums + (size_t)i * Fs + x0, lane, acc);
        }
        float eacc = 0.0f;
        for (uint32_t c = c0; c < c1; ++c) eacc += __ldcg(s.chunk_epart + c);
        if (lane == 0) sums_e[i] = eacc;
    }
}

// apply_nsvd_deltas (src/tsvdx4p.rs:341-385) of summed deltas: sums [I, Fs],
// sums_e [I] and, with the per-day terms, the fixed-point yfeat_day sums.
template <int VPL>
__global__ void __launch_bounds__(kThreads) k_y_apply_sums(DeviceState s, EpochParams p,
                                                           const float* __restrict__ sums,
                                                           const float* __restrict__ sums_e,
                                                           const long long* __restrict__ dyd) {
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs;
    const uint32_t warps = gridDim.x * kWarps;
    for (uint32_t i = blockIdx.x * kWarps + (threadIdx.x >> 5); i < s.n_items; i += warps) {
        const uint64_t ncnt = s.item_off[i + 1] - s.item_off[i];
        if (ncnt == 0) continue;
        const float scale = p.nsvd_norm_exp == 0.0f ? 1.0f : powf((float)ncnt, p.nsvd_norm_exp);
        for (uint32_t x0 = 0; x0 < Fs; x0 += 32 * VPL) {
            float acc[VPL], y[VPL];
            Row<VPL>::load_cg(sums + (size_t)i * Fs + x0, lane, acc);
            Row<VPL>::load_cg(s.yfeat + (size_t)i * Fs + x0, lane, y);
#pragma unroll
            for (int v = 0; v < VPL; ++v) y[v] = y[v] - p.lr_y * (acc[v] / scale + p.reg_y * y[v]);
            Row<VPL>::store(s.yfeat + (size_t)i * Fs + x0, lane, y);
            if (dyd) {
                float yd[VPL];
                Row<VPL>::load_cg(s.yfeat_day + (size_t)i * Fs + x0, lane, yd);
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    const float d = (float)((double)__ldcg(dyd + (size_t)i * Fs + x0 + Row<VPL>::elem(lane, v)) /
                                            kDydScale);
                    yd[v] = yd[v] - p.lr_yd * (d / scale + p.reg_yd * yd[v]);
                }
                Row<VPL>::store(s.yfeat_day + (size_t)i * Fs + x0, lane, yd);
            }
        }
        if (lane == 0) s.ybias[i] = s.ybias[i] - p.lr_yb * (__ldcg(sums_e + i) / scale);
    }
}

// ---------------------------------------------------------------------------
// Rows above 2,048 columns (tsvd_wide.cu has those of more than 256; the tsvdx4 jobs
// go up to 4800 factors, tsvdx4p up to 16000): rows
// of Fs = 256 k columns. A warp's unit keeps its own rows in global memory
// (they are private to it, and each lane reads back only what it wrote) and
// takes each rating in two passes over 256-column slices: the dot product,
// then the updates. Per element the arithmetic is that of the narrow kernels.
// ---------------------------------------------------------------------------
constexpr int kWV = 8;                   // values per lane in a slice
constexpr uint32_t kSlice = 32 * kWV;    // columns per slice

__global__ void __launch_bounds__(kThreads) k_user_strat_wide(DeviceState s, EpochParams p,
                                                              const uint32_t* __restrict__ order, uint32_t n_work) {
    using R8 = Row<kWV>;
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs, T = s.T, NF = s.NF;
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
        float* pu_row = s.ufeat + (size_t)u * Fs;
        float* p2_row = s.ufeat2 + (size_t)u * Fs;
        float* su_row = s.ycache + (size_t)u * Fs;
        float* sq_row = s.g_user + (size_t)u * Fs;  // the NSVD1 error sum, then the user's gradient
        float sub;
        if (p.use_ycache) {
            sub = __ldcg(s.ycache_bias + u);
        } else {
            sub = 0.0f;
            for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
                float su[kWV], sb = 0.0f;
#pragma unroll
                for (int v = 0; v < kWV; ++v) su[v] = 0.0f;
                const Rec* rr = s.rec + start;
                gather_rows8<kWV>(s.yfeat + c0, c0 == 0 ? s.ybias : nullptr, Fs, end - start,
                                  [&](uint64_t q) { return rec_id(__ldg(&rr[q].key)); }, lane, su, sb);
                if (p.full_su) {
                    const uint32_t* pp = s.pr_item + ps;
                    gather_rows8<kWV>(s.yfeat + c0, c0 == 0 ? s.ybias : nullptr, Fs, pe - ps,
                                      [&](uint64_t q) { return __ldg(pp + q); }, lane, su, sb);
                }
#pragma unroll
                for (int v = 0; v < kWV; ++v) su[v] = su[v] / norm;
                R8::store(su_row + c0, lane, su);
                if (c0 == 0) sub = sb / norm;
            }
            if (lane == 0) s.ycache_bias[u] = sub;
        }
        {
            const float z[kWV] = {};
            for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) R8::store(sq_row + c0, lane, z);
        }
        float ub = __ldcg(s.ubias + u), al = __ldcg(s.alpha_u + u), cuu = __ldcg(s.cu + u);
        float bb0 = lane < (int)T ? __ldcg(s.but_bin + (size_t)u * T + lane) : 0.0f;
        float bb1 = lane + 32 < (int)T ? __ldcg(s.but_bin + (size_t)u * T + 32 + lane) : 0.0f;
        float sum_err = 0.0f;
        const float gb = s.gbias;
        for (uint64_t base = start; base < end; base += 32) {
            const uint32_t cnt = (uint32_t)(end - base < 32 ? end - base : 32);
            Rec mine{};
            if (lane < (int)cnt) mine = load_rec(s.rec + base + lane);
            for (uint32_t j = 0; j < cnt; ++j) {
                const Rec r = shfl_rec(mine, j);
                const uint32_t i = rec_id(r.key), tb = rec_tbin(r.key);
                const bool hud = r.ud < s.n_ud;
                const float* qe_row = s.qe0 + (size_t)i * Fs;  // q_i + q^f_{i,0} (low_memory: bin 0)
                const float ib = __ldg(s.ibias + i);
                const float bit = __ldg(s.bit_bin + (size_t)i * T + tb);
                const float ibf = __ldg(s.ibias_freq + (size_t)i * NF);
                float bud = 0.0f;
                if (lane == 0 && hud) bud = s.ubias_day[r.ud];
                bud = __shfl_sync(kFull, bud, 0);
                const float ct = hud ? __ldg(s.cut + r.ud) : 0.0f;
                const float but = __shfl_sync(kFull, tb < 32 ? bb0 : bb1, tb & 31);
                const float dv = r.dev;
                const float bu_t = ub + but + al * dv + bud + sub;
                const float bi_t = ib + bit + ibf;
                const float cu_t = cuu + ct;
                float part = 0.0f;
                for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
                    float qe[kWV], pu[kWV], su[kWV], p2[kWV];
                    R8::load_nc(qe_row + c0, lane, qe);
                    R8::load_cg(pu_row + c0, lane, pu);
                    R8::load_cg(su_row + c0, lane, su);
                    R8::load_cg(p2_row + c0, lane, p2);
#pragma unroll
                    for (int v = 0; v < kWV; ++v) part += qe[v] * ((pu[v] + su[v]) + dv * p2[v]);
                }
                const float dot = warp_sum(part);
                const float err = gb + bu_t + bi_t * cu_t + dot - r.res;
                ub -= p.lr_ub * err;
                {
                    const float nb = but - p.lr_tu * err;
                    if (lane == (int)(tb & 31)) {
                        if (tb < 32) bb0 = nb;
                        else bb1 = nb;
                    }
                }
                al -= p.lr_ta * err * dv;
                if (lane == 0 && hud) s.ubias_day[r.ud] = bud - p.lr_ubd * err;
                cuu -= p.lr_cu * (err * bi_t + p.reg_cu * (cuu - 1.0f));
                sum_err += err;
                for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
                    float qev[kWV], pu[kWV], p2[kWV], sq[kWV];
                    R8::load_nc(qe_row + c0, lane, qev);
                    R8::load_cg(pu_row + c0, lane, pu);
                    R8::load_cg(p2_row + c0, lane, p2);
                    R8::load_cg(sq_row + c0, lane, sq);
#pragma unroll
                    for (int v = 0; v < kWV; ++v) {
                        const float qe = qev[v];
                        const float pk = pu[v], p2k = p2[v];
                        sq[v] += err * qe;
                        pu[v] = pk - p.lr_u * (err * qe + p.reg_u * pk);
                        p2[v] = p2k - p.lr_u2 * (err * qe * dv + p.reg_u2 * p2k);
                    }
                    R8::store(pu_row + c0, lane, pu);
                    R8::store(p2_row + c0, lane, p2);
                    R8::store(sq_row + c0, lane, sq);
                }
            }
        }
        if (lane == 0) {
            s.ubias[u] = ub;
            s.alpha_u[u] = al;
            s.cu[u] = cuu;
        }
        if (lane < (int)T) s.but_bin[(size_t)u * T + lane] = bb0;
        if (lane + 32 < (int)T) s.but_bin[(size_t)u * T + 32 + lane] = bb1;
        for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
            float g[kWV];
            R8::load_cg(sq_row + c0, lane, g);
#pragma unroll
            for (int v = 0; v < kWV; ++v) g[v] = g[v] / norm;
            R8::store(sq_row + c0, lane, g);
        }
        if (lane == 0) s.e_user[u] = sum_err / norm;
    }
}

// Item stratum for rows above 2,048 columns: one warp per item, the item's q and q^f rows in
// global memory, every item on the one-warp chain.
__global__ void __launch_bounds__(kThreads) k_item_wide(DeviceState s, EpochParams p) {
    using R8 = Row<kWV>;
    const int lane = threadIdx.x & 31;
    const uint32_t Fs = s.Fs, NF = s.NF;
    const float gb = s.gbias;
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&s.counters[2], 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= s.n_item_work) break;
        const uint32_t i = s.item_work[k];
        const uint64_t a = s.item_off[i], b = s.item_off[i + 1];
        if (a == b) continue;
        float* q_row = s.ifeat + (size_t)i * Fs;
        float* qf_base = s.ifeat_freq + (size_t)i * NF * Fs;
        ItemState st = load_item_state(s, i, lane);
        for (uint64_t base = a; base < b; base += 32) {
            const uint32_t cnt = (uint32_t)(b - base < 32 ? b - base : 32);
            Rec mine{};
            float bu_l = 0.0f, cu_l = 0.0f;
            if (lane < (int)cnt) {
                mine = load_rec(s.irec + base + lane);
                user_scalars(s, mine, bu_l, cu_l);
            }
            for (uint32_t j = 0; j < cnt; ++j) {
                const Rec r = shfl_rec(mine, j);
                const uint32_t u = rec_id(r.key), tb = rec_tbin(r.key), fb = rec_fbin(r.key);
                const float bu_t = __shfl_sync(kFull, bu_l, j), cu_t = __shfl_sync(kFull, cu_l, j);
                const float* pyc_row = s.pyc + (size_t)u * Fs;
                const float* p2_row = s.ufeat2 + (size_t)u * Fs;
                float* qf_row = qf_base + (size_t)fb * Fs;
                const float bit = __shfl_sync(kFull, tb < 32 ? st.bt0 : st.bt1, tb & 31);
                const float ibf = __shfl_sync(kFull, fb < 32 ? st.bf0 : st.bf1, fb & 31);
                const float bi_t = st.ib + bit + ibf;
                float part = 0.0f;
                for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
                    float x[kWV], y[kWV], q[kWV], qf[kWV];
                    R8::load_nc(pyc_row + c0, lane, x);
                    R8::load_nc(p2_row + c0, lane, y);
                    R8::load_cg(q_row + c0, lane, q);
                    R8::load_cg(qf_row + c0, lane, qf);
#pragma unroll
                    for (int v = 0; v < kWV; ++v) part += (x[v] + r.dev * y[v]) * (q[v] + qf[v]);
                }
                const float dot = warp_sum(part);
                const float err = gb + bu_t + bi_t * cu_t + dot - r.res;
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
                for (uint32_t c0 = 0; c0 < Fs; c0 += kSlice) {
                    float x[kWV], y[kWV], q[kWV], qf[kWV];
                    R8::load_nc(pyc_row + c0, lane, x);
                    R8::load_nc(p2_row + c0, lane, y);
                    R8::load_cg(q_row + c0, lane, q);
                    R8::load_cg(qf_row + c0, lane, qf);
#pragma unroll
                    for (int v = 0; v < kWV; ++v) {
                        const float pev = x[v] + r.dev * y[v];
                        const float qi = q[v];
                        q[v] = qi - p.lr_i * (err * pev + p.reg_i * qi);
                        qf[v] = qf[v] - p.lr_iqf * (err * pev + p.reg_iqf * qf[v]);
                    }
                    R8::store(q_row + c0, lane, q);
                    R8::store(qf_row + c0, lane, qf);
                }
            }
        }
        store_item_state(s, i, lane, st);
    }
}

// The wide strata's launches.
void launch_user_wide(tsvd_model* m, const EpochParams& p, const uint32_t* work, uint32_t n) {
    if (wide_pairs_fit(m->d.Fs)) {
        launch_user_wide_pairs(m, m->d, p, work, n);
        return;
    }
    k_user_strat_wide<<<persistent_grid(k_user_strat_wide, 0), kThreads, 0, m->stream>>>(m->d, p, work, n);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

void launch_item_wide(tsvd_model* m, const DeviceState& s, const EpochParams& p) {
    if (wide_pairs_fit(s.Fs)) {
        launch_item_wide_pairs(m, s, p);
        return;
    }
    k_item_wide<<<persistent_grid(k_item_wide, 0), kThreads, 0, m->stream>>>(s, p);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

void strat_launch_wide(tsvd_model* m, const EpochParams& p) {
    const DeviceState& s = m->d;
    make_qe0(m, false);
    {
        ProfScope ps(m, "user_pass_stratified");
        launch_user_wide(m, p, s.user_work, s.n_users);
    }
    {
        ProfScope ps(m, "y_apply");
        y_partial_passes<kWV>(m, s, 0, s.n_users);
        k_y_combine<kWV><<<ceil_div(s.n_items, kWarps), kThreads, 0, m->stream>>>(s, p);
        TSVD_CUDA(cudaGetLastError());
        m->launches++;
    }
    launch_rebuild_ycache(m, s.pyc);
    {
        ProfScope ps(m, "item_pass");
        launch_item_wide(m, s, p);
    }
}

void make_qe0(tsvd_model* m, bool bf16) {
    const DeviceState& s = m->d;
    if (!s.qe0) return;
    const unsigned grid = (unsigned)std::min<uint64_t>(((uint64_t)s.n_items * s.Fs + 255) / 256, 148ull * 32);
    k_make_qe0<<<grid, 256, 0, m->stream>>>(s.ifeat, s.ifeat_freq, s.n_items, s.Fs, s.NF, bf16, s.qe0);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

void to_bf16(tsvd_model* m, const float* src, uint64_t rows, uint64_t src_stride, void* dst) {
    const uint32_t Fs = m->d.Fs;
    const unsigned grid = (unsigned)std::min<uint64_t>((rows * Fs + 255) / 256, 148ull * 32);
    k_to_bf16<<<grid, 256, 0, m->stream>>>(src, rows, Fs, src_stride, (__nv_bfloat16*)dst);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

// One stratified epoch (Tsvdx4pModel::fit_epoch, src/tsvdx4p.rs:815-822):
// user stratum, NSVD1 delta sums and apply, ycache (and ycache_day) rebuild,
// item stratum.
template <int VPL, bool BF, bool BFU, bool DAY>
void strat_launch(tsvd_model* m, const EpochParams& p, const Bf16Copies& bf) {
    DeviceState s = m->d;
    if (DAY) TSVD_CUDA(cudaMemsetAsync(s.dyd_fix, 0, (size_t)s.n_items * s.Fs * 8, m->stream));
    if (!DAY) make_qe0(m, BF);
    {
        ProfScope ps(m, "user_pass_stratified");
        if constexpr (DAY) {
            launch_user_days(m, s, p, s.user_work, s.n_users);
        } else {
            launch_user_stratum(m, s, p, bf, s.user_work, s.n_users);
        }
    }
    {
        ProfScope ps(m, "y_apply");
        y_partial_passes<VPL>(m, s, 0, s.n_users);
        k_y_combine<VPL><<<ceil_div(s.n_items, kWarps), kThreads, 0, m->stream>>>(s, p);
        TSVD_CUDA(cudaGetLastError());
        m->launches++;
    }
    if (BF) to_bf16(m, s.yfeat, s.n_items, s.Fs, m->m_bf_yfeat.p);
    launch_rebuild_ycache(m, s.pyc);
    if (DAY) rebuild_ycache_day(m);
    if (BFU) {
        ProfScope ps(m, "bf16_copies");
        to_bf16(m, s.pyc, s.n_users, s.Fs, m->m_bf_pyc.p);
        to_bf16(m, s.ufeat2, s.n_users, s.Fs, m->m_bf_ufeat2.p);
    }
    {
        ProfScope ps(m, "item_pass");
        launch_item_stratum(m, s, p, bf);
    }
}

// Standard init of a set of users: p_u rows given (host-drawn), the rest as
// TxModel::new leaves it (src/tx.rs:600-648).
__global__ void k_reset_users(DeviceState s, const uint32_t* __restrict__ users, uint32_t n,
                              const float* __restrict__ prow) {
    const uint32_t w = blockIdx.x;
    if (w >= n) return;
    const uint32_t u = users[w];
    for (uint32_t c = threadIdx.x; c < s.Fs; c += blockDim.x) {
        s.ufeat[(size_t)u * s.Fs + c] = prow[(size_t)w * s.Fs + c];
        s.ufeat2[(size_t)u * s.Fs + c] = 0.0f;
    }
    for (uint32_t b = threadIdx.x; b < s.T; b += blockDim.x) s.but_bin[(size_t)u * s.T + b] = 0.0f;
    for (uint64_t d = s.ud_start[u] + threadIdx.x; d < s.ud_start[u + 1]; d += blockDim.x) s.ubias_day[d] = 0.0f;
    if (threadIdx.x == 0) {
        s.ubias[u] = 0.0f;
        s.alpha_u[u] = 0.0f;
        s.cu[u] = 1.0f;
    }
}

// (With the per-day terms the fold-in's yfeat_day deltas land in dyd_fix,
// which the next stratified epoch clears before its user stratum.)
void foldin_launch(tsvd_model* m, const EpochParams& p, const uint32_t* d_users, uint32_t n) {
    if (m->d.dyd_fix) {
        launch_user_days(m, m->d, p, d_users, n);
    } else {
        make_qe0(m, false);
        launch_user_stratum(m, m->d, p, Bf16Copies{}, d_users, n);
    }
}

// ---------------------------------------------------------------------------
// A sharded run's steps (one process per GPU, users and items in contiguous
// blocks): the user stratum of a user block with the block's NSVD1 delta sums,
// the apply of the summed deltas with the cache rebuild, and the item stratum
// of an item block. The exchanges between them are the caller's collectives.
// ---------------------------------------------------------------------------
template <int VPL, bool DAY>
void shard_user_launch(tsvd_model* m, const EpochParams& p, const uint32_t* work, uint32_t n, uint32_t u_lo,
                       uint32_t u_hi, float* sums, float* sums_e) {
    const DeviceState& s = m->d;
    if (!DAY) make_qe0(m, false);
    {
        ProfScope ps(m, "user_pass_stratified");
        if (s.Fs > kSlice) {
            launch_user_wide(m, p, work, n);
        } else {
            if constexpr (DAY) {
                launch_user_days(m, s, p, work, n);
            } else {
                launch_user_stratum(m, s, p, Bf16Copies{}, work, n);
            }
        }
    }
    ProfScope ps(m, "y_apply");
    y_partial_passes<VPL>(m, s, u_lo, u_hi);
    k_y_block_sums<VPL><<<ceil_div(s.n_items, kWarps), kThreads, 0, m->stream>>>(s, sums, sums_e);
    TSVD_CUDA(cudaGetLastError());
    m->launches++;
}

void shard_item_launch(tsvd_model* m, const EpochParams& p, const uint32_t* work, uint32_t n) {
    DeviceState s = m->d;
    s.item_work = work;
    s.n_item_work = n;
    ProfScope ps(m, "item_pass");
    if (s.Fs > kSlice) {
        launch_item_wide(m, s, p);
    } else {
        launch_item_stratum(m, s, p, Bf16Copies{});
    }
}

// Units lo..hi-1 of a count table, heaviest first (ties by id).
std::vector<uint32_t> block_work(uint32_t lo, uint32_t hi, const std::function<uint64_t(uint32_t)>& count) {
    std::vector<uint32_t> w(hi - lo);
    std::iota(w.begin(), w.end(), lo);
    std::stable_sort(w.begin(), w.end(), [&](uint32_t a, uint32_t b) { return count(a) > count(b); });
    return w;
}

void upload_work(tsvd_model* m, const std::vector<uint32_t>& w) {
    if (m->m_shard_work.bytes < std::max<size_t>(w.size(), 1) * 4) m->m_shard_work.alloc(std::max<size_t>(w.size(), 1) * 4);
    if (!w.empty())
        TSVD_CUDA(cudaMemcpyAsync(m->m_shard_work.p, w.data(), w.size() * 4, cudaMemcpyHostToDevice, m->stream));
    TSVD_CUDA(cudaStreamSynchronize(m->stream));  // `w` leaves scope
}

void check_shardable(const tsvd_model* m) {
    if (m->opts.schedule != TSVD_SCHED_STRATIFIED || m->opts.precision != TSVD_PREC_FP32)
        throw Error(TSVD_ERR_UNSUPPORTED, "a sharded run needs the stratified schedule with FP32 reads");
}

}  // namespace

void stratified_epoch(tsvd_model* m, const EpochParams& p) {
    const DeviceState& s = m->d;
    const int prec = m->opts.precision;
    Bf16Copies bf{};
    if (prec >= TSVD_PREC_BF16_READ) {
        ProfScope ps(m, "bf16_copies");
        to_bf16(m, s.yfeat, s.n_items, s.Fs, m->m_bf_yfeat.p);
        bf.yfeat = m->m_bf_yfeat.as<__nv_bfloat16>();
    }
    if (prec >= TSVD_PREC_BF16_READ_ALL) {
        bf.pyc = m->m_bf_pyc.as<__nv_bfloat16>();
        bf.ufeat2 = m->m_bf_ufeat2.as<__nv_bfloat16>();
    }
    const int vpl = (int)(s.Fs / 32);
    if (s.Fs > kSlice) {  // n_feat > 256: low_memory, FP32
        strat_launch_wide(m, p);
    } else if (s.dyd_fix) {  // low_memory = false (FP32 only)
        TSVD_DISPATCH(vpl, (strat_launch<V, false, false, true>(m, p, bf)));
    } else if (prec == TSVD_PREC_FP32) {
        TSVD_DISPATCH(vpl, (strat_launch<V, false, false, false>(m, p, bf)));
    } else if (prec == TSVD_PREC_BF16_READ) {
        TSVD_DISPATCH(vpl, (strat_launch<V, true, false, false>(m, p, bf)));
    } else {
        TSVD_DISPATCH(vpl, (strat_launch<V, true, true, false>(m, p, bf)));
    }
}

}  // namespace tsvd

// ---------------------------------------------------------------------------
// Fold-in and user reset entry points.
// ---------------------------------------------------------------------------
extern "C" int tsvd_foldin(tsvd_model* m, const uint32_t* users, uint64_t n, uint32_t passes) {
    using namespace tsvd;
    if (!m || (!users && n)) return TSVD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(m->mu);
    return guarded(m, [&] {
        if (n == 0 || passes == 0) return;
        if (n >= (1ull << 32)) throw Error(TSVD_ERR_INVALID, "too many users");
        if (m->d.Fs > kSlice) throw Error(TSVD_ERR_UNSUPPORTED, "fold-in is built for n_feat up to 256");
        for (uint64_t k = 0; k < n; ++k)
            if (users[k] >= m->d.n_users) throw Error(TSVD_ERR_INVALID, "user out of range");
        TSVD_CUDA(cudaSetDevice(m->device));
        DevMem du;
        du.alloc(n * 4);
        TSVD_CUDA(cudaMemcpyAsync(du.p, users, n * 4, cudaMemcpyHostToDevice, m->stream));
        if (!m->ycache_valid) {
            launch_rebuild_ycache(m);
        }
        EpochParams p = make_params(m);
        p.use_ycache = m->cfg.full_su ? 1 : 0;
        for (uint32_t k = 0; k < passes; ++k) {
            TSVD_CUDA(cudaMemsetAsync(m->d.counters, 0, 64, m->stream));
            foldin_launch(m, p, du.as<uint32_t>(), (uint32_t)n);
        }
        TSVD_CUDA(cudaStreamSynchronize(m->stream));
    });
}

extern "C" int tsvd_reset_users(tsvd_model* m, const uint32_t* users, uint64_t n, uint64_t seed) {
    using namespace tsvd;
    if (!m || (!users && n)) return TSVD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(m->mu);
    return guarded(m, [&] {
        if (n == 0) return;
        for (uint64_t k = 0; k < n; ++k)
            if (users[k] >= m->d.n_users) throw Error(TSVD_ERR_INVALID, "user out of range");
        TSVD_CUDA(cudaSetDevice(m->device));
        const uint32_t Fs = m->d.Fs, F = m->d.F;
        std::vector<float> h((size_t)n * Fs, 0.0f);
        ChaCha12Stream g(seed);
        fill_normal_rows(g, m->cfg.sigma_u, n, F, h.data(), Fs);
        DevMem du, dp;
        du.alloc(n * 4);
        dp.alloc(h.size() * 4);
        TSVD_CUDA(cudaMemcpyAsync(du.p, users, n * 4, cudaMemcpyHostToDevice, m->stream));
        TSVD_CUDA(cudaMemcpyAsync(dp.p, h.data(), h.size() * 4, cudaMemcpyHostToDevice, m->stream));
        k_reset_users<<<(unsigned)n, 128, 0, m->stream>>>(m->d, du.as<uint32_t>(), (uint32_t)n, dp.as<float>());
        TSVD_CUDA(cudaGetLastError());
        TSVD_CUDA(cudaStreamSynchronize(m->stream));
    });
}

// ---------------------------------------------------------------------------
// Sharded-run entry points.
// ---------------------------------------------------------------------------
extern "C" int tsvd_shard_user_block(tsvd_model* m, uint64_t epoch, uint32_t u_lo, uint32_t u_hi, float* d_sums,
                                     float* d_sums_e, int64_t* d_dyd) {
    using namespace tsvd;
    if (!m) return TSVD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(m->mu);
    return guarded(m, [&] {
        check_shardable(m);
        if (epoch == 0) throw Error(TSVD_ERR_INVALID, "epoch is 1-based");
        if (u_lo > u_hi || u_hi > m->d.n_users) throw Error(TSVD_ERR_INVALID, "user block out of range");
        if (!d_sums || !d_sums_e || (m->d.dyd_fix && !d_dyd))
            throw Error(TSVD_ERR_INVALID, "null delta buffer");
        use_device(m);
        const DeviceState& s = m->d;
        if (epoch == m->cfg.reset_u_epoch) {
            TSVD_CUDA(cudaMemsetAsync(s.ufeat, 0, m->m_ufeat.bytes, m->stream));
            TSVD_CUDA(cudaMemsetAsync(s.ufeat2, 0, m->m_ufeat2.bytes, m->stream));
        }
        TSVD_CUDA(cudaMemsetAsync(s.counters, 0, 64, m->stream));
        std::vector<uint32_t> w = block_work(u_lo, u_hi, [&](uint32_t u) { return (uint64_t)m->h_user_cnt[u]; });
        upload_work(m, w);
        EpochParams p = make_params(m);
        p.use_ycache = (m->cfg.full_su && m->ycache_valid) ? 1 : 0;
        if (s.dyd_fix) TSVD_CUDA(cudaMemsetAsync(s.dyd_fix, 0, (size_t)s.n_items * s.Fs * 8, m->stream));
        const int vpl = (int)std::min<uint32_t>(s.Fs / 32, 8);
        if (s.dyd_fix) {
            TSVD_DISPATCH(vpl, (shard_user_launch<V, true>(m, p, m->m_shard_work.as<uint32_t>(), (uint32_t)w.size(),
                                                          u_lo, u_hi, d_sums, d_sums_e)));
            TSVD_CUDA(cudaMemcpyAsync(d_dyd, s.dyd_fix, (size_t)s.n_items * s.Fs * 8, cudaMemcpyDeviceToDevice,
                                      m->stream));
        } else {
            TSVD_DISPATCH(vpl, (shard_user_launch<V, false>(m, p, m->m_shard_work.as<uint32_t>(), (uint32_t)w.size(),
                                                           u_lo, u_hi, d_sums, d_sums_e)));
        }
        m->ycache_valid = false;  // the ycache rows of the block's users were rewritten from the current y
        TSVD_CUDA(cudaStreamSynchronize(m->stream));
    });
}

extern "C" int tsvd_shard_apply(tsvd_model* m, const float* d_sums, const float* d_sums_e, const int64_t* d_dyd) {
    using namespace tsvd;
    if (!m) return TSVD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(m->mu);
    return guarded(m, [&] {
        check_shardable(m);
        if (!d_sums || !d_sums_e || (m->d.dyd_fix && !d_dyd)) throw Error(TSVD_ERR_INVALID, "null delta buffer");
        use_device(m);
        const DeviceState& s = m->d;
        const EpochParams p = make_params(m);
        const int vpl = (int)std::min<uint32_t>(s.Fs / 32, 8);
        {
            ProfScope ps(m, "y_apply");
            TSVD_DISPATCH(vpl, (k_y_apply_sums<V><<<ceil_div(s.n_items, kWarps), kThreads, 0, m->stream>>>(
                                   s, p, d_sums, d_sums_e, s.dyd_fix ? (const long long*)d_dyd : nullptr)));
            TSVD_CUDA(cudaGetLastError());
            m->launches++;
        }
        launch_rebuild_ycache(m, s.pyc);
        rebuild_ycache_day(m);
        TSVD_CUDA(cudaStreamSynchronize(m->stream));
    });
}

extern "C" int tsvd_shard_item_block(tsvd_model* m, uint32_t i_lo, uint32_t i_hi) {
    using namespace tsvd;
    if (!m) return TSVD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(m->mu);
    return guarded(m, [&] {
        check_shardable(m);
        if (i_lo > i_hi || i_hi > m->d.n_items) throw Error(TSVD_ERR_INVALID, "item block out of range");
        use_device(m);
        const DeviceState& s = m->d;
        if (m->h_item_off.empty()) {
            m->h_item_off.resize((size_t)s.n_items + 1);
            TSVD_CUDA(cudaMemcpy(m->h_item_off.data(), s.item_off, m->h_item_off.size() * 8, cudaMemcpyDeviceToHost));
        }
        TSVD_CUDA(cudaMemsetAsync(s.counters, 0, 64, m->stream));
        std::vector<uint32_t> w =
            block_work(i_lo, i_hi, [&](uint32_t i) { return m->h_item_off[i + 1] - m->h_item_off[i]; });
        upload_work(m, w);
        const EpochParams p = make_params(m);
        shard_item_launch(m, p, m->m_shard_work.as<uint32_t>(), (uint32_t)w.size());
        TSVD_CUDA(cudaStreamSynchronize(m->stream));
        finish_epoch(m);
    });
}
