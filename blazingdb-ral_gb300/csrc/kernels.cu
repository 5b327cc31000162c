// kernels.cu — ahead-of-time kernels of the expression path (nvcc, sm_103a).
//
//   ral_count_valid      null_count recount (GDFColumn.cu:519-529 uses cudf's
//                        gdf_count_nonzero_mask)
//   ral_gather_*         materialize_column (ColumnManipulation.cu:26-150): data
//                        gather plus validity gather with ballot-built words
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_rt.cuh"
#include "kernels.h"
#include "engine.h"

namespace ral {

namespace {

__global__ void count_valid_kernel(const ral_u32* __restrict__ valid, ral_i64 n, unsigned long long* out) {
    const ral_i64 words = (n + 31) >> 5;
    ral_u64 acc = 0;
    for (ral_i64 w = (ral_i64)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += (ral_i64)gridDim.x * blockDim.x) {
        ral_u32 v = __ldg(valid + w);
        const ral_i64 rem = n - (w << 5);
        if (rem < 32) v &= (1u << rem) - 1u;
        acc += __popc(v);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    __shared__ ral_u64 red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        ral_u64 t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
        if (t) atomicAdd(out, (unsigned long long)t);
    }
}

// One thread per output row; a warp builds each 32-row output validity word
// with a ballot, so there is no read-modify-write of shared words.
template <typename E, typename I>
__global__ void gather_kernel(const E* __restrict__ in, const ral_u32* __restrict__ in_valid, ral_i64 n_in,
                              const I* __restrict__ idx, ral_i64 n_out, E* __restrict__ out,
                              ral_u32* __restrict__ out_valid, unsigned long long* valid_count) {
    ral_u64 cnt = 0;
    const ral_i64 stride = (ral_i64)gridDim.x * blockDim.x;
    const ral_i64 n_round = (n_out + 31) & ~(ral_i64)31;
    for (ral_i64 i = (ral_i64)blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += stride) {
        bool bit = false;
        if (i < n_out) {
            const ral_i64 j = (ral_i64)idx[i];
            if (j >= 0 && j < n_in) {
                out[i] = in[j];
                bit = in_valid ? ((__ldg(in_valid + (j >> 5)) >> (j & 31)) & 1u) : true;
            }
        }
        if (out_valid) {
            const ral_u32 word = __ballot_sync(0xffffffffu, bit);
            if ((threadIdx.x & 31) == 0) {
                out_valid[i >> 5] = word;
                cnt += __popc(word);
            }
        }
    }
    if (valid_count) {
        for (int off = 16; off > 0; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
        if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(valid_count, (unsigned long long)cnt);
    }
}

template <typename E>
cudaError_t gather_by_index(const void* in, const uint32_t* in_valid, int64_t n_in, const void* idx, int idx_width,
                            int64_t n_out,
                            void* out, uint32_t* out_valid, unsigned long long* valid_count, cudaStream_t st) {
    const int threads = 256;
    int64_t blocks = (n_out + threads - 1) / threads;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    const E* i_ = (const E*)in;
    E* o_ = (E*)out;
    switch (idx_width) {
    case 1: gather_kernel<E, int8_t><<<(int)blocks, threads, 0, st>>>(i_, in_valid, n_in, (const int8_t*)idx, n_out, o_, out_valid, valid_count); break;
    case 2: gather_kernel<E, int16_t><<<(int)blocks, threads, 0, st>>>(i_, in_valid, n_in, (const int16_t*)idx, n_out, o_, out_valid, valid_count); break;
    case 4: gather_kernel<E, int32_t><<<(int)blocks, threads, 0, st>>>(i_, in_valid, n_in, (const int32_t*)idx, n_out, o_, out_valid, valid_count); break;
    case 8: gather_kernel<E, int64_t><<<(int)blocks, threads, 0, st>>>(i_, in_valid, n_in, (const int64_t*)idx, n_out, o_, out_valid, valid_count); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}


// ---- every column of a frame gathered by one index column -----------------------------------
// A warp takes 128 consecutive output rows per step; lane t handles rows base + t + 32 k (k < 4),
// so each k is one coalesced index load, one coalesced store per column and one ballot-built
// validity word per nullable column, and every lane has eight independent loads in flight per
// column (four elements, four mask words).
//
// Two orders, chosen per launch from a sample of the index (every block computes the same choice):
// * clustered indices (a filter's kept rows, a sorted join side): row-major -- a step gathers every
//   column, so the index is read once and each column's nearby rows share cache lines;
// * scattered indices (an order-by permutation, a hash join): column-major -- the whole grid
//   gathers one column before the next.  Each column's random reads then stay within its own
//   span, and its validity mask (n/8 bytes) stays in L2 instead of competing with every other
//   column's mask; measured on six columns of 200M rows by a permutation, row-major took 48.7 ms
//   against 33.4 ms for six one-column passes.  The index is re-read per column (4 B per row).
// In the column-major order element loads are marked evict-first (`ld.global.cs`): a scattered
// element is read once, and the masks are what L2 should keep (clustered rows share lines, so the
// row-major order loads them normally).
constexpr int kGatherRowsPerLane = 4;
constexpr int kGatherSamples = 64;          // index samples of 32 consecutive rows
constexpr ral_u32 kGatherClusterSpan = 1u << 16;  // a sample spanning fewer input rows is clustered

template <typename I>
__device__ __forceinline__ ral_i64 ral_load_index(const void* idx, ral_i64 i) {
    return (ral_i64)__ldcs(reinterpret_cast<const I*>(idx) + i);
}

__device__ __forceinline__ ral_i64 ral_index_at(const GatherColumnsParams& P, ral_i64 i) {
    switch (P.idx_width) {
    case 1: return ral_load_index<int8_t>(P.idx, i);
    case 2: return ral_load_index<int16_t>(P.idx, i);
    case 4: return ral_load_index<int32_t>(P.idx, i);
    default: return ral_load_index<long long>(P.idx, i);
    }
}

// One column's step: the four element loads and the four validity-word loads are all issued before
// any is used (their values feed only the stores and ballots after them).
template <typename E, bool kScattered>
__device__ __forceinline__ unsigned ral_gather_k(const GatherColumn& c, const ral_i64 (&j)[kGatherRowsPerLane],
                                                 const bool (&ok)[kGatherRowsPerLane], ral_i64 base, int lane,
                                                 ral_i64 n_out) {
    const E* __restrict__ in = reinterpret_cast<const E*>(c.in);
    E* __restrict__ out = reinterpret_cast<E*>(c.out);
    const ral_u32* __restrict__ iv = c.in_valid;
    E v[kGatherRowsPerLane];
    ral_u32 w[kGatherRowsPerLane];
#pragma unroll
    for (int k = 0; k < kGatherRowsPerLane; ++k) {
        v[k] = ok[k] ? (kScattered ? __ldcs(in + j[k]) : __ldg(in + j[k])) : E(0);
        w[k] = ok[k] ? (iv ? __ldg(iv + (j[k] >> 5)) : 0xffffffffu) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kGatherRowsPerLane; ++k)
        if (ok[k]) __stcs(out + base + lane + 32 * k, v[k]);
    unsigned cnt = 0;
    if (c.out_valid) {
#pragma unroll
        for (int k = 0; k < kGatherRowsPerLane; ++k) {
            const bool bit = (w[k] >> (j[k] & 31)) & 1u;
            const ral_u32 word = __ballot_sync(0xffffffffu, bit);
            // word k covers rows base + 32 k .. +31; lane k writes it (masks are padded to 64
            // bytes, so a partial last word stays inside the allocation)
            if (lane == k && base + 32 * k < n_out) c.out_valid[(base >> 5) + k] = word;
            cnt += __popc(word);
        }
    }
    return cnt;
}

template <bool kScattered>
__device__ __forceinline__ unsigned ral_gather_column_step(const GatherColumn& col, const ral_i64 (&j)[kGatherRowsPerLane],
                                                           const bool (&ok)[kGatherRowsPerLane], ral_i64 base,
                                                           int lane, ral_i64 n_out) {
    switch (col.width) {
    case 1: return ral_gather_k<int8_t, kScattered>(col, j, ok, base, lane, n_out);
    case 2: return ral_gather_k<short, kScattered>(col, j, ok, base, lane, n_out);
    case 4: return ral_gather_k<int, kScattered>(col, j, ok, base, lane, n_out);
    default: return ral_gather_k<long long, kScattered>(col, j, ok, base, lane, n_out);
    }
}

__device__ __forceinline__ void ral_step_indices(const GatherColumnsParams& P, ral_i64 base, int lane,
                                                 ral_i64 (&j)[kGatherRowsPerLane], bool (&ok)[kGatherRowsPerLane]) {
#pragma unroll
    for (int k = 0; k < kGatherRowsPerLane; ++k) {
        const ral_i64 i = base + lane + 32 * k;
        j[k] = i < P.n_out ? ral_index_at(P, i) : -1;
        ok[k] = j[k] >= 0 && j[k] < P.n_in;
    }
}

// Clustered samples among the 8 that warp `warp` (0 .. 7) tests, their loads in flight together (one
// sample after the other took 25 us per launch); kept out of line so that its registers do not add to
// the gather loops'.
__device__ __noinline__ int ral_gather_votes(const GatherColumnsParams& P, int warp, int lane) {
    ral_u32 lo[kGatherSamples / 8], hi[kGatherSamples / 8];
#pragma unroll
    for (int q = 0; q < kGatherSamples / 8; ++q) {
        const ral_i64 at = (P.n_out - 32) / (kGatherSamples - 1) * (warp * (kGatherSamples / 8) + q);
        const ral_i64 j = ral_index_at(P, at + lane);
        const bool in = j >= 0 && j < P.n_in;  // rows are 32-bit: an index inside the input fits
        lo[q] = in ? (ral_u32)j : 0xffffffffu;
        hi[q] = in ? (ral_u32)j : 0u;
    }
    int votes = 0;
#pragma unroll
    for (int q = 0; q < kGatherSamples / 8; ++q) {
        const ral_u32 a = __reduce_min_sync(0xffffffffu, lo[q]), b = __reduce_max_sync(0xffffffffu, hi[q]);
        votes += (b < a || b - a < kGatherClusterSpan) ? 1 : 0;
    }
    return votes;
}

// 48 registers, five resident blocks of 256 threads per SM (a bound of six spills registers in the
// gather loops).
__global__ void __launch_bounds__(256, 5) gather_columns_kernel(const __grid_constant__ GatherColumnsParams P) {
    if (P.scattered && (*P.scattered != 0) != (P.only_scattered != 0)) return;
    __shared__ unsigned long long s_cnt[kMaxGatherColumns];
    __shared__ int s_clustered;
    for (int c = threadIdx.x; c < P.num_columns; c += blockDim.x) s_cnt[c] = 0;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // the order: each warp tests 8 samples of 32 consecutive indices (the same samples in every block); a
    // sample is clustered when its in-range indices span fewer than
    // kGatherClusterSpan input rows; a launch is clustered when at least half its samples are
    if (threadIdx.x == 0) s_clustered = 0;
    __syncthreads();
    if (!P.scattered && P.num_columns > 1 && P.n_out >= 32 * kGatherSamples) {
        const int votes = ral_gather_votes(P, warp, lane);
        if (lane == 0) atomicAdd(&s_clustered, votes);
    }
    __syncthreads();
    const bool row_major = P.num_columns == 1 || (P.scattered ? P.only_scattered == 0 : P.n_out < 32 * kGatherSamples || 2 * s_clustered >= kGatherSamples);
    const ral_i64 step_rows = 32 * kGatherRowsPerLane;
    const ral_i64 nsteps = (P.n_out + step_rows - 1) / step_rows;
    const ral_i64 gwarp = ((ral_i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const ral_i64 nwarp = ((ral_i64)gridDim.x * blockDim.x) >> 5;
    if (row_major) {
        for (ral_i64 s = gwarp; s < nsteps; s += nwarp) {
            const ral_i64 base = s * step_rows;
            ral_i64 j[kGatherRowsPerLane];
            bool ok[kGatherRowsPerLane];
            ral_step_indices(P, base, lane, j, ok);
            for (int c = 0; c < P.num_columns; ++c) {
                const unsigned cnt = ral_gather_column_step<false>(P.col[c], j, ok, base, lane, P.n_out);
                if (lane == 0 && cnt) atomicAdd(&s_cnt[c], (unsigned long long)cnt);
            }
        }
    } else {
        for (int c = 0; c < P.num_columns; ++c) {
            unsigned long long cc = 0;
            for (ral_i64 s = gwarp; s < nsteps; s += nwarp) {
                const ral_i64 base = s * step_rows;
                ral_i64 j[kGatherRowsPerLane];
                bool ok[kGatherRowsPerLane];
                ral_step_indices(P, base, lane, j, ok);
                cc += ral_gather_column_step<true>(P.col[c], j, ok, base, lane, P.n_out);
            }
            if (lane == 0 && cc) atomicAdd(&s_cnt[c], cc);
        }
    }
    __syncthreads();
    if (P.valid_counts)
        for (int c = threadIdx.x; c < P.num_columns; c += blockDim.x)
            if (s_cnt[c]) atomicAdd(P.valid_counts + c, s_cnt[c]);
}

__global__ void __launch_bounds__(256) gather_probe_kernel(const __grid_constant__ GatherColumnsParams P, int32_t* scattered) {
    __shared__ int s_votes;
    if (threadIdx.x == 0) s_votes = 0;
    __syncthreads();
    const int votes = ral_gather_votes(P, threadIdx.x >> 5, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_votes, votes);
    __syncthreads();
    if (threadIdx.x == 0) *scattered = 2 * s_votes >= kGatherSamples ? 0 : 1;
}

// ---- single-pass stream compaction (decoupled look-back) ---------------------------------
// Tile = 256 threads x 16 rows; the look-back is ral_lookback (device_rt.cuh).

__global__ void __launch_bounds__(256) compact_stencil_kernel(const int8_t* __restrict__ stencil,
                                                              const ral_u32* __restrict__ valid, ral_i64 n,
                                                              int32_t* __restrict__ out, ral_u64* scratch) {
    __shared__ ral_u32 s_tile;
    __shared__ ral_u32 s_warp[8];
    __shared__ ral_u64 s_prefix;
    ral_u64* status = scratch + 3;
    const ral_i64 ntiles = (n + kCompactTileRows - 1) / kCompactTileRows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec_ok = (((uintptr_t)stencil) & 15) == 0;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd((unsigned int*)scratch, 1u);
        __syncthreads();
        const ral_i64 tile = s_tile;
        if (tile >= ntiles) break;
        const ral_i64 r0 = tile * kCompactTileRows + (ral_i64)threadIdx.x * 16;
        ral_u32 keep = 0;
        if (r0 + 16 <= n && vec_ok) {
            const uint4 v = __ldcs(reinterpret_cast<const uint4*>(stencil + r0));
            const ral_u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 16; k++) keep |= (((w[k >> 2] >> (8 * (k & 3))) & 0xffu) != 0u ? 1u : 0u) << k;
        } else {
            for (int k = 0; k < 16; k++)
                if (r0 + k < n && stencil[r0 + k] != 0) keep |= 1u << k;
        }
        if (valid && r0 < n) keep &= (__ldg(valid + (r0 >> 5)) >> (r0 & 31)) & 0xffffu;
        const ral_u32 cnt = __popc(keep);
        ral_u32 incl = cnt;
        for (int off = 1; off < 32; off <<= 1) {
            const ral_u32 t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            ral_u32 wv = lane < 8 ? s_warp[lane] : 0;
            ral_u32 wi = wv;
            for (int off = 1; off < 8; off <<= 1) {
                const ral_u32 t = __shfl_up_sync(0xffffffffu, wi, off);
                if (lane >= off) wi += t;
            }
            const ral_u32 total = __shfl_sync(0xffffffffu, wi, 7);
            const ral_u64 excl = ral_lookback(status, tile, total, scratch + 1);
            if (lane < 8) s_warp[lane] = wi - wv;
            if (lane == 0) {
                s_prefix = excl;
                if (tile == ntiles - 1) scratch[2] = excl + total;
            }
        }
        __syncthreads();
        ral_u64 pos = s_prefix + s_warp[warp] + (incl - cnt);
        while (keep) {
            const int k = __ffs(keep) - 1;
            keep &= keep - 1;
            out[pos++] = (int32_t)(r0 + k);
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_count_valid(const uint32_t* valid, int64_t n, unsigned long long* out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    int64_t words = (n + 31) / 32;
    int64_t blocks = (words + threads - 1) / threads;
    if (blocks > 152 * 8) blocks = 152 * 8;
    count_valid_kernel<<<(int)blocks, threads, 0, st>>>(valid, n, out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_compact_stencil(const int8_t* stencil, const uint32_t* stencil_valid, int64_t n, int32_t* out_idx,
                                   unsigned long long* scratch, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int dev = 0, sms = 1, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, compact_stencil_kernel, 256, 0);
    if (per_sm < 1) per_sm = 1;
    const int64_t tiles = (n + kCompactTileRows - 1) / kCompactTileRows;
    int64_t grid = std::min<int64_t>(tiles, (int64_t)sms * per_sm);
    compact_stencil_kernel<<<(int)grid, 256, 0, st>>>(stencil, stencil_valid, n, out_idx, (ral_u64*)scratch);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gather(int width, const void* in, const uint32_t* in_valid, int64_t n_in, const void* idx,
                          int idx_width, int64_t n_out, void* out, uint32_t* out_valid, unsigned long long* valid_count,
                          cudaStream_t st) {
    if (n_out <= 0) return cudaSuccess;
    switch (width) {
    case 1: return gather_by_index<int8_t>(in, in_valid, n_in, idx, idx_width, n_out, out, out_valid, valid_count, st);
    case 2: return gather_by_index<int16_t>(in, in_valid, n_in, idx, idx_width, n_out, out, out_valid, valid_count, st);
    case 4: return gather_by_index<int32_t>(in, in_valid, n_in, idx, idx_width, n_out, out, out_valid, valid_count, st);
    case 8: return gather_by_index<int64_t>(in, in_valid, n_in, idx, idx_width, n_out, out, out_valid, valid_count, st);
    default: return cudaErrorInvalidValue;
    }
}

namespace {
__global__ void category_insert_kernel(int32_t* __restrict__ codes, ral_i64 n, int32_t pos) {
    const ral_i64 stride = (ral_i64)gridDim.x * blockDim.x;
    for (ral_i64 i = (ral_i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        if (codes[i] >= pos) codes[i] += 1;
}
__global__ void category_remap_kernel(int32_t* __restrict__ codes, ral_i64 n, const int32_t* __restrict__ table,
                                      int32_t table_n) {
    const ral_i64 stride = (ral_i64)gridDim.x * blockDim.x;
    for (ral_i64 i = (ral_i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int32_t c = codes[i];
        if (c >= 0 && c < table_n) codes[i] = __ldg(table + c);
    }
}
}  // namespace

// ---- line index of a delimited text buffer ---------------------------------------------------
// Tile t of 64 KiB in 16 steps of 4 KiB: in step k, thread j reads bytes [16 j, 16 j + 16) of the
// step (one 16-byte load where the buffer allows it; a warp's loads are one contiguous 512 bytes),
// so a step's terminators come out in order from a block-wide scan of the threads' counts, and the
// steps in turn.

__device__ __forceinline__ ral_u32 ral_text_term_bits(const char* data, int64_t n, int64_t at, char term) {
    ral_u32 bits = 0;
    if (at + 16 <= n && ((uintptr_t)(data + at) & 15) == 0) {
        const uint4 v = __ldcs(reinterpret_cast<const uint4*>(data + at));
        const ral_u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 16; ++k)
            bits |= ((ral_u32)(((w[k >> 2] >> (8 * (k & 3))) & 0xffu) == (ral_u32)(unsigned char)term)) << k;
    } else {
        for (int k = 0; k < 16; ++k)
            if (at + k < n && data[at + k] == term) bits |= 1u << k;
    }
    return bits;
}

__global__ void __launch_bounds__(256) text_term_count_kernel(const char* __restrict__ data, int64_t n, char term,
                                                              ral_u32* __restrict__ counts) {
    const int64_t tile = blockIdx.x;
    ral_u32 c = 0;
#pragma unroll 4
    for (int k = 0; k < (int)(kTextTileBytes / kTextStepBytes); ++k)
        c += __popc(ral_text_term_bits(data, n, tile * kTextTileBytes + k * kTextStepBytes + 16 * (int64_t)threadIdx.x, term));
    __shared__ ral_u32 s_w[8];
    const ral_u32 wsum = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = wsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        ral_u32 t = 0;
        for (int w = 0; w < 8; ++w) t += s_w[w];
        counts[tile] = t;
    }
}

__global__ void __launch_bounds__(1024) exclusive_scan_u32_kernel(const ral_u32* __restrict__ counts, int64_t m,
                                                                  unsigned long long* __restrict__ offsets) {
    __shared__ unsigned long long s_w[32];
    __shared__ unsigned long long s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t base = 0; base < m; base += 1024) {
        const int64_t i = base + threadIdx.x;
        const unsigned long long v = i < m ? counts[i] : 0ull;
        unsigned long long inc = v;
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = s_w[lane];
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xffffffffu, w, off);
                if (lane >= off) w += t;
            }
            s_w[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const unsigned long long carry = s_carry;
        const unsigned long long before = (warp ? s_w[warp - 1] : 0ull) + inc - v;
        if (i < m) offsets[i] = carry + before;
        __syncthreads();
        if (threadIdx.x == 0) s_carry = carry + s_w[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) offsets[m] = s_carry;
}

__global__ void __launch_bounds__(256) text_term_positions_kernel(const char* __restrict__ data, int64_t n, char term,
                                                                  const unsigned long long* __restrict__ offsets,
                                                                  long long* __restrict__ ends) {
    const int64_t tile = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ ral_u32 s_w[2][8];
    unsigned long long base = offsets[tile];
    for (int k = 0; k < (int)(kTextTileBytes / kTextStepBytes); ++k) {
        const int64_t at = tile * kTextTileBytes + k * kTextStepBytes + 16 * (int64_t)threadIdx.x;
        if (tile * kTextTileBytes + k * kTextStepBytes >= n) break;  // block-uniform
        ral_u32 bits = ral_text_term_bits(data, n, at, term);
        const ral_u32 c = __popc(bits);
        ral_u32 inc = c;
        for (int off = 1; off < 32; off <<= 1) {
            const ral_u32 t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        if (lane == 31) s_w[k & 1][warp] = inc;  // double-buffered: no barrier between a step's reads and the next step's writes
        __syncthreads();
        ral_u32 before = inc - c, step_total = 0;
        for (int w = 0; w < 8; ++w) {
            const ral_u32 x = s_w[k & 1][w];
            if (w < warp) before += x;
            step_total += x;
        }
        unsigned long long q = base + before;
        for (; bits; bits &= bits - 1u) ends[q++] = at + __ffs(bits) - 1;
        base += step_total;
    }
}

// One block: the tile holding the k-th terminator from the tiles' offsets (or the first one), then
// steps of 4 KiB until it is reached.
__global__ void __launch_bounds__(256) text_skip_kernel(const char* __restrict__ data, int64_t n, char term, int64_t k,
                                                        const unsigned long long* __restrict__ offsets, int64_t tiles,
                                                        unsigned long long* __restrict__ out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ ral_u32 s_w[2][8];
    int64_t at0 = 0, seen = 0;
    if (offsets) {
        int64_t a = 0, b = tiles;  // the last tile with fewer than k terminators before it
        while (b - a > 1) {
            const int64_t m = (a + b) / 2;
            if ((int64_t)offsets[m] < k) a = m;
            else b = m;
        }
        at0 = a * kTextTileBytes;
        seen = (int64_t)offsets[a];
    }
    for (int i = 0; at0 < n; ++i, at0 += kTextStepBytes) {
        const int64_t at = at0 + 16 * (int64_t)threadIdx.x;
        ral_u32 bits = ral_text_term_bits(data, n, at, term);
        const ral_u32 c = __popc(bits);
        ral_u32 inc = c;
        for (int off = 1; off < 32; off <<= 1) {
            const ral_u32 t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        if (lane == 31) s_w[i & 1][warp] = inc;
        __syncthreads();
        int64_t before = seen + inc - c, total = seen;
        for (int w = 0; w < 8; ++w) {
            const ral_u32 x = s_w[i & 1][w];
            if (w < warp) before += x;
            total += x;
        }
        if (before < k && before + c >= k) {
            for (int64_t j = before + 1; j < k; ++j) bits &= bits - 1u;
            *out = (unsigned long long)(at + __ffs(bits));
        }
        if (total >= k) return;  // block-uniform
        seen = total;
    }
    if (threadIdx.x == 0) *out = (unsigned long long)n;
}

__global__ void __launch_bounds__(256) text_present_count_kernel(const char* __restrict__ data, int64_t n,
                                                                 const long long* __restrict__ ends, int64_t nterm,
                                                                 int64_t lines, int64_t skip,
                                                                 unsigned long long* count) {
    ral_u32 c = 0;
    for (int64_t i = skip + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < lines;
         i += (int64_t)gridDim.x * blockDim.x) {
        const long long s = i == 0 ? 0 : ends[i - 1] + 1;
        long long e = i < nterm ? ends[i] : n;
        if (e > s && data[e - 1] == '\r') --e;
        c += e > s ? 1u : 0u;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
}

cudaError_t launch_text_present_count(const char* data, int64_t n, const long long* ends, int64_t nterm, int64_t lines,
                                      int64_t skip, unsigned long long* count, cudaStream_t st) {
    if (lines <= skip) return cudaSuccess;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((lines - skip + 255) / 256, 152 * 8));
    text_present_count_kernel<<<(int)blocks, 256, 0, st>>>(data, n, ends, nterm, lines, skip, count);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_text_term_counts(const char* data, int64_t n, char term, uint32_t* counts, cudaStream_t st) {
    const int64_t tiles = text_tiles(n);
    if (tiles <= 0) return cudaSuccess;
    if (tiles > 0x7fffffffll) return cudaErrorInvalidValue;
    text_term_count_kernel<<<(unsigned)tiles, 256, 0, st>>>(data, n, term, counts);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_exclusive_scan_u32(const uint32_t* counts, int64_t tiles, unsigned long long* offsets,
                                      cudaStream_t st) {
    exclusive_scan_u32_kernel<<<1, 1024, 0, st>>>(counts, tiles, offsets);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_text_skip(const char* data, int64_t n, char term, int64_t k, const unsigned long long* offsets,
                             unsigned long long* out, cudaStream_t st) {
    text_skip_kernel<<<1, 256, 0, st>>>(data, n, term, k, offsets, text_tiles(n), out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_text_term_positions(const char* data, int64_t n, char term, const unsigned long long* offsets,
                                       long long* ends, cudaStream_t st) {
    const int64_t tiles = text_tiles(n);
    if (tiles <= 0) return cudaSuccess;
    if (tiles > 0x7fffffffll) return cudaErrorInvalidValue;
    text_term_positions_kernel<<<(unsigned)tiles, 256, 0, st>>>(data, n, term, offsets, ends);
    note_launch();
    return cudaGetLastError();
}

// ---- Parquet data pages ----------------------------------------------------------------------
// A required column's page is its values back to back; an optional column's page starts with the
// 4-byte length of its definition levels (bit width 1) in the RLE / bit-packed hybrid (a run
// header varint h: h odd -> h >> 1 groups of 8 bit-packed levels, h even -> h >> 1 repeats of the
// next byte's level), then the values of the present rows only.  Two kernels:
//  * levels, one block per optional page: the run headers become a table (a batch of up to kPqRuns
//    runs at a time) and the block writes the validity words from it, 32 rows per thread, counting
//    the present rows of each 8192-row item; the counts become each item's first value index;
//  * values, one block per 8192-row item of a page: a required page copies its rows' values; an
//    optional page ranks each row among its item's present rows (a block scan of the validity
//    words' popcounts) and fetches its value.


constexpr int kPqRuns = 1024;
constexpr int kPqWindow = 12288;  // level bytes of a page staged in shared memory at a time

// An 8- or 4-byte little-endian value at base + i * w, where base has any alignment: two aligned
// loads and a funnel shift (the second load stays inside the 8-byte word holding the value's last
// byte, so it never leaves the buffer).
__device__ __forceinline__ unsigned long long ral_pq_value(const uint8_t* base, int64_t i, int w) {
    const uintptr_t a = (uintptr_t)(base + i * w);
    if (w == 8) {
        const int s = (int)(a & 7);
        const unsigned long long* q = reinterpret_cast<const unsigned long long*>(a - s);
        const unsigned long long lo = q[0];
        return s ? (lo >> (8 * s)) | (q[1] << (64 - 8 * s)) : lo;
    }
    const int s = (int)(a & 3);
    const ral_u32* q = reinterpret_cast<const ral_u32*>(a - s);
    const ral_u32 lo = q[0];
    return s ? (ral_u32)((lo >> (8 * s)) | (q[1] << (32 - 8 * s))) : lo;
}

__device__ __forceinline__ void ral_pq_store(void* base, int64_t i, int w, unsigned long long v) {
    if (w == 8) reinterpret_cast<unsigned long long*>(base)[i] = v;
    else reinterpret_cast<unsigned int*>(base)[i] = (unsigned int)v;
}

// A run header of a level stream: rows of the run, the byte its bits (or its level) start at, how many
// bytes those are, and the bytes from the header to the next one.
struct LevelRun {
    int pay, after, hop;
    int len;       // clamped to 2^30
    bool packed, ok;
};
// The run whose header starts at byte `at` of the staged stream bytes w (which go on for 8 bytes past any
// header); the stream ends at byte `end`.
__device__ __forceinline__ LevelRun ral_level_run(const uint8_t* w, int at, int end) {
    LevelRun r{0, 0, INT_MAX, 0, false, false};
    const ral_u32 b0 = w[at], b1 = w[at + 1];
    ral_u32 n = b0 & 0x7fu;
    if (!(b0 & 0x80u)) {
        r.pay = at + 1;
    } else if (!(b1 & 0x80u)) {
        n |= b1 << 7;
        r.pay = at + 2;
    } else {
        unsigned long long h = n | (b1 & 0x7fu) << 7;
        int shift = 14, p = at + 2;
        for (;; shift += 7) {
            if (shift > 35) return r;
            const unsigned long long b = w[p++];
            h |= (b & 0x7f) << shift;
            if (!(b & 0x80)) break;
        }
        r.pay = p;
        n = (ral_u32)min(h, (1ull << 31) - 2 + (h & 1));  // a run's groups or rows, clamped
    }
    r.packed = (n & 1u) != 0u;
    n >>= 1;
    r.len = (int)(r.packed ? min(n, 1u << 27) * 8u : n);
    // a header or a run past the stream's end does not read
    r.ok = r.pay <= end && (r.packed ? n <= (ral_u32)(end - r.pay) : r.pay < end);
    if (r.ok) {
        r.after = r.packed ? (int)n : 1;
        r.hop = r.pay - at + r.after;
    }
    return r;
}

constexpr int kLevelThreads = 1024;

// Rows [rel0, rel1) of a required page of PLAIN values, by 256 threads of which this one is t.
__device__ __forceinline__ void ral_pq_plain_rows(const ParquetPage& pg, const ParquetColumnOut& col, int rel0, int rel1, int t) {
    const int lane = t & 31, warp = t >> 5, w = col.width;
    const uint8_t* const vals = (const uint8_t*)pg.data + pg.values_off;
    // Every row has its value (the page's length is checked on the host).  The lanes of a
    // warp take consecutive rows: each loads the aligned word where its value starts and
    // takes the next word from the lane after it (the last lane of the run loads it), so a
    // warp reads one contiguous aligned span whatever the values' alignment.
    const uintptr_t va = (uintptr_t)vals;
    if (w == 8) {
        // 16-byte words: lane l takes rows 2m, 2m + 1 (m = the warp's pair + l), bytes
        // [s + 16m, s + 16m + 16) past the aligned base: word m and, when s > 0, word m + 1
        // from the next lane (the last lane of the run loads it, when its values reach it)
        const int s16 = (int)(va & 15);
        const int k = s16 >> 2, f = (s16 & 3) * 8;
        const uint4* q = reinterpret_cast<const uint4*>(va - s16);
        unsigned long long* out = reinterpret_cast<unsigned long long*>(col.data) + pg.row_start;
#pragma unroll 2
        for (int m0 = (rel0 >> 1) + 32 * warp; 2 * m0 < rel1; m0 += 256) {
            const int m = m0 + lane;
            const int r = 2 * m;
            const bool in = r < rel1;
            const uint4 a = in ? q[m] : make_uint4(0u, 0u, 0u, 0u);
            uint4 b;
            b.x = __shfl_down_sync(0xffffffffu, a.x, 1);
            b.y = __shfl_down_sync(0xffffffffu, a.y, 1);
            b.z = __shfl_down_sync(0xffffffffu, a.z, 1);
            b.w = __shfl_down_sync(0xffffffffu, a.w, 1);
            const bool two = r + 1 < rel1;
            if (in && (lane == 31 || r + 2 >= rel1) && s16 + (two ? 16 : 8) > 16) b = q[m + 1];
            ral_u32 o0, o1, o2, o3;
            switch (k) {  // uniform over the page
            case 0: o0 = a.x; o1 = a.y; o2 = a.z; o3 = a.w; if (f) { o0 = __funnelshift_r(a.x, a.y, f); o1 = __funnelshift_r(a.y, a.z, f); o2 = __funnelshift_r(a.z, a.w, f); o3 = __funnelshift_r(a.w, b.x, f); } break;
            case 1: o0 = __funnelshift_r(a.y, a.z, f); o1 = __funnelshift_r(a.z, a.w, f); o2 = __funnelshift_r(a.w, b.x, f); o3 = __funnelshift_r(b.x, b.y, f); break;
            case 2: o0 = __funnelshift_r(a.z, a.w, f); o1 = __funnelshift_r(a.w, b.x, f); o2 = __funnelshift_r(b.x, b.y, f); o3 = __funnelshift_r(b.y, b.z, f); break;
            default: o0 = __funnelshift_r(a.w, b.x, f); o1 = __funnelshift_r(b.x, b.y, f); o2 = __funnelshift_r(b.y, b.z, f); o3 = __funnelshift_r(b.z, b.w, f); break;
            }
            if (in) out[r] = (unsigned long long)o1 << 32 | o0;
            if (two) out[r + 1] = (unsigned long long)o3 << 32 | o2;
        }
    } else {
        const int sh = (int)(va & 3) * 8;
        const ral_u32* q = reinterpret_cast<const ral_u32*>(va - (va & 3));
        ral_u32* out = reinterpret_cast<ral_u32*>(col.data) + pg.row_start;
#pragma unroll 4
        for (int r0 = rel0 + 32 * warp; r0 < rel1; r0 += 256) {
            const int r = r0 + lane;
            const bool in = r < rel1;
            const ral_u32 lo = in ? q[r] : 0u;
            ral_u32 nx = __shfl_down_sync(0xffffffffu, lo, 1);
            if (sh && in && (lane == 31 || r + 1 >= rel1)) nx = q[r + 1];
            if (in) out[r] = sh ? (lo >> sh) | (nx << (32 - sh)) : lo;
        }
    }
}

// The page of an item: the last one whose first item is at or before it.
__device__ __forceinline__ int ral_pq_page_of(const ParquetDecodeParams& P, int item) {
    int a = P.page_lo, b = P.page_hi - 1;
    while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (P.pages[m].item0 <= item) a = m;
        else b = m - 1;
    }
    return a;
}

// A block beyond the pages' own of a 1024-thread kernel: the items 4 k .. 4 k + 3 of every plain_every-th one,
// of which it writes those of required PLAIN pages.
__device__ __forceinline__ void ral_pq_plain_block(const ParquetDecodeParams& P, int k) {
    const int item = P.item_lo + (4 * k + (int)(threadIdx.x >> 8)) * P.plain_every;
    if (item >= P.item_hi) return;
    const ParquetPage pg = P.pages[ral_pq_page_of(P, item)];
    if (pg.optional || pg.dict_count > 0) return;
    const int rel0 = (item - pg.item0) * kParquetItemRows;
    ral_pq_plain_rows(pg, P.out[pg.column], rel0, min(rel0 + kParquetItemRows, pg.rows), threadIdx.x & 255);
}

// One block per optional page.  The run headers form a chain of which only the start is known.  Every
// byte of a 12 KiB window of the stream is read as if a header started there, by all threads, which
// leaves the bytes to the next one; thread 0 then only adds hops (some 45 cycles a run), and the runs it
// lists are read a thread each into a table, from which every thread writes 32 rows' validity at a time.
// Bound: the latency of a page's steps (one block a page).  24 pages of 131,072 rows, 12 of them with 3%
// nulls (15.6 KB, 600 runs): 46 us, 72 with 256 threads a block and 141 when thread 0 read every header
// itself.  (Composing the hops of 32-byte segments in parallel and writing bits a run a thread measured
// 205 us.)  These few blocks leave the device and the link to the file idle: further blocks write the values
// of required PLAIN pages, which wait for nothing (the scan with these pages 198 -> 183 us).
__global__ void __launch_bounds__(kLevelThreads) parquet_levels_kernel(const __grid_constant__ ParquetDecodeParams P) {
    __shared__ ral_u32 s_lw[kPqWindow / 4 + 8];
    __shared__ uint16_t s_hop[kPqWindow];  // per byte of the window: the bytes to the next header if one starts there
    __shared__ uint16_t s_start[kPqRuns];
    __shared__ int s_row[kPqRuns + 1];
    __shared__ int s_info[kPqRuns];  // bit-packed: byte offset of the run's levels; RLE: the level
    __shared__ unsigned char s_kind[kPqRuns];
    __shared__ int s_n, s_new, s_bad, s_emit, s_emit_end, s_done;
    __shared__ long long s_pos, s_w[kLevelThreads / 32];
    if ((int)blockIdx.x >= P.page_hi - P.page_lo) {
        ral_pq_plain_block(P, (int)blockIdx.x - (P.page_hi - P.page_lo));
        return;
    }
    const ParquetPage pg = P.pages[P.page_lo + blockIdx.x];
    if (!pg.optional || pg.rows <= 0) return;
    const ParquetColumnOut col = P.out[pg.column];
    const uint8_t* const lev = (const uint8_t*)pg.data + pg.lev_off;
    const int lev_bytes = pg.levels;
    if (threadIdx.x == 0) {
        s_pos = 0;
        s_n = 0;
        s_row[0] = 0;
        s_bad = 0;
        s_emit = 0;
        s_done = 0;
    }
    __syncthreads();
    const int words = (pg.rows + 31) >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int w0 = -1, off = 0, have = 0;  // the window: stream bytes [w0, w0 + have) are staged
    auto lb = [&](long long p) -> unsigned long long {
        const int o = (int)p - w0;
        return o >= 0 && o < have ? reinterpret_cast<const uint8_t*>(s_lw)[off + o] : (p < lev_bytes ? lev[p] : 0u);
    };
    while (true) {
        const int pos = (int)s_pos;
        if (w0 < 0 || pos >= w0 + kPqWindow) {
            // the next window, and the bytes of a header that starts at its end; aligned words that stay
            // inside the page's data or the buffer's 16-byte padding
            w0 = pos;
            off = (int)((uintptr_t)(lev + w0) & 3);
            have = min(kPqWindow + 16, lev_bytes - w0);
            for (int i = threadIdx.x; i < (off + have + 3) >> 2; i += kLevelThreads)
                s_lw[i] = reinterpret_cast<const ral_u32*>(lev + w0 - off)[i];
            __syncthreads();
            for (int p = threadIdx.x; p < min(kPqWindow, have); p += kLevelThreads)
                s_hop[p] = (uint16_t)min(ral_level_run(reinterpret_cast<const uint8_t*>(s_lw) + off, p, lev_bytes - w0).hop, 0xffff);
            __syncthreads();
        }
        const uint8_t* const sb = reinterpret_cast<const uint8_t*>(s_lw) + off;
        // thread 0 follows the headers, whose runs are then read a thread each
        const int carried = s_n, size = min(kPqWindow, have);
        if (threadIdx.x == 0) {
            int p = pos - w0, k = 0;
            const int room = kPqRuns - carried;
            while (k < room && p < size) {
                s_start[k++] = (uint16_t)p;
                p += s_hop[p];
            }
            s_new = k;
        }
        __syncthreads();
        const int fresh = s_new;
        LevelRun run[kPqRuns / kLevelThreads];
        long long rows = 0;  // this thread's runs' rows, and (above 2^40) how many of them have some
#pragma unroll
        for (int q = 0; q < kPqRuns / kLevelThreads; ++q) {
            const int k = (int)threadIdx.x * (kPqRuns / kLevelThreads) + q;
            run[q].len = 0;
            if (k < fresh) {
                run[q] = ral_level_run(sb, s_start[k], lev_bytes - w0);
                if (k == fresh - 1) s_pos = run[q].ok ? (long long)w0 + run[q].pay + run[q].after : -1;
                if (!run[q].ok) run[q].len = 0;
            }
            rows += run[q].len + ((long long)(run[q].len > 0) << 44);
        }
        long long inc = rows;
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        long long before = inc - rows, total = 0;
        for (int w = 0; w < kLevelThreads / 32; ++w) {
            if (w < warp) before += s_w[w];
            total += s_w[w];
        }
        long long at = s_row[carried] + (before & ((1ll << 44) - 1));
        int slot = carried + (int)(before >> 44);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kPqRuns / kLevelThreads; ++q) {
            if (run[q].len <= 0) continue;  // runs of no rows are left out
            s_kind[slot] = run[q].packed ? 1 : 0;
            s_info[slot] = run[q].packed ? w0 + run[q].pay : sb[run[q].pay] & 1;
            at += run[q].len;
            s_row[++slot] = (int)min(at, (long long)pg.rows);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_n = carried + (int)(total >> 44);
            const int row = s_row[s_n];
            // a header that does not read (it is the last listed), or a stream that ends, before the rows
            if (row < pg.rows && (s_pos < 0 || fresh == 0)) s_bad = 1;
            // whole words covered by the table (all of them once the page's rows are)
            s_emit_end = row >= pg.rows ? words : (row >> 5);
        }
        __syncthreads();
        if (s_bad) break;
        const int n = s_n, e0 = s_emit, e1 = s_emit_end;
        for (int k0 = e0; k0 < e1; k0 += kLevelThreads) {
            const int k = k0 + (int)threadIdx.x;
            ral_u32 X = 0;
            if (k < e1) {
                const int r0 = 32 * k, r1 = min(r0 + 32, pg.rows);
                int a = 0, b = n - 1;  // the last run starting at or before r0
                while (a < b) {
                    const int m = (a + b + 1) >> 1;
                    if (s_row[m] <= r0) a = m;
                    else b = m - 1;
                }
                for (int r = r0; r < r1; ++a) {
                    const int re = min(s_row[a + 1], r1);
                    const int len = re - r;
                    const ral_u32 m = len == 32 ? 0xffffffffu : ((1u << len) - 1u);
                    ral_u32 bits;
                    if (s_kind[a]) {
                        const int bo = r - s_row[a];
                        const long long p = s_info[a] + (bo >> 3);
                        const unsigned long long v = lb(p) | lb(p + 1) << 8 | lb(p + 2) << 16 | lb(p + 3) << 24 | lb(p + 4) << 32;
                        bits = (ral_u32)(v >> (bo & 7)) & m;
                    } else {
                        bits = s_info[a] ? m : 0u;
                    }
                    X |= bits << (r - r0);
                    r = re;
                }
            }
            // present rows per item (a warp's 32 words lie in at most two items)
            const int first = (k0 + 32 * warp) >> 8;
            const ral_u32 c = __popc(X);
            const ral_u32 ca = (k >> 8) == first ? c : 0u;
            const ral_u32 sa = __reduce_add_sync(0xffffffffu, ca);
            const ral_u32 sb2 = __reduce_add_sync(0xffffffffu, c - ca);
            if (lane == 0) {
                if (sa) atomicAdd(P.item_base + pg.item0 + first, sa);
                if (sb2) atomicAdd(P.item_base + pg.item0 + first + 1, sb2);
            }
            if (X) {
                const int64_t g = pg.row_start + 32 * (int64_t)k;
                const int sh = (int)(g & 31);
                ral_u32* const vw = col.valid + (g >> 5);
                if (sh == 0 && 32 * k + 32 <= pg.rows) {
                    *vw = X;  // the word holds rows of this page only
                } else {
                    atomicOr(vw, X << sh);
                    const ral_u32 hi = sh ? X >> (32 - sh) : 0u;
                    if (hi) atomicOr(vw + 1, hi);
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_emit = e1;
            if (e1 >= words) {
                s_done = 1;
            } else {
                // carry the runs that reach into the first word not written yet
                const int from = 32 * e1;
                int a = 0, b = n;  // the first run that ends after it
                while (a < b) {
                    const int m = (a + b) >> 1;
                    if (s_row[m + 1] <= from) a = m + 1;
                    else b = m;
                }
                for (int j = a; j <= n; ++j) {
                    s_row[j - a] = s_row[j];
                    if (j < n) {
                        s_kind[j - a] = s_kind[j];
                        s_info[j - a] = s_info[j];
                    }
                }
                s_n = n - a;
            }
        }
        __syncthreads();
        if (s_done) break;
    }
    if (s_bad) {
        if (threadIdx.x == 0) {
            atomicAdd(P.status, 1ull);
            P.page_present[P.page_lo + blockIdx.x] = 0u;  // no indices are read for this page
        }
        return;
    }
    if (warp == 0) {
        // item counts -> each item's first value index; the page's values must cover them
        const int items = (pg.rows + kParquetItemRows - 1) / kParquetItemRows;
        ral_u32 run = 0;
        for (int i = 0; i < items; i += 32) {
            const ral_u32 c = i + lane < items ? __ldcg(P.item_base + pg.item0 + i + lane) : 0u;
            ral_u32 inc = c;
            for (int o = 1; o < 32; o <<= 1) {
                const ral_u32 t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (i + lane < items) P.item_base[pg.item0 + i + lane] = run + inc - c;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane) return;
        // PLAIN values must cover the present rows (a dictionary page's indices are checked by
        // their own kernel)
        const int64_t nvals = (pg.data_bytes - (int64_t)pg.values_off) / col.width;
        if (pg.dict_count == 0 && (int64_t)run > nvals) atomicAdd(P.status, 1ull);
        P.page_present[P.page_lo + blockIdx.x] = run;
        if (run) atomicAdd(P.status + 1 + pg.column, (unsigned long long)run);
    }
}

__global__ void __launch_bounds__(256) parquet_values_kernel(const __grid_constant__ ParquetDecodeParams P) {
    __shared__ ral_u32 s_word[256];
    __shared__ ral_u32 s_base[256];
    __shared__ ral_u32 s_wsum[8];
    const int item = P.item_lo + (int)blockIdx.x;
    const ParquetPage pg = P.pages[ral_pq_page_of(P, item)];
    const ParquetColumnOut col = P.out[pg.column];
    const int w = col.width;
    const int rel0 = (item - pg.item0) * kParquetItemRows;
    const int rel1 = min(rel0 + kParquetItemRows, pg.rows);
    const int64_t lo = pg.values_off;
    const uint8_t* const vals = (const uint8_t*)pg.data + lo;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (pg.dict_count > 0 && !pg.optional) {
        // a dictionary-encoded required page: row r's entry is idx[idx0 + r] (checked in range)
        const uint8_t* const dict = (const uint8_t*)pg.dict;
        const uint32_t* const ix = P.idx + pg.idx0;
        // four rows at a time: their index loads, then their entries' loads, are in flight together
        for (int r0 = rel0 + (int)threadIdx.x; r0 < rel1; r0 += 1024) {
            uint32_t k[4];
            unsigned long long x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = r0 + 256 * u < rel1 ? ix[r0 + 256 * u] : 0xffffffffu;
#pragma unroll
            for (int u = 0; u < 4; ++u)  // in range unless the page was malformed (then reported)
                x[u] = k[u] < (uint32_t)pg.dict_count ? ral_pq_value(dict, k[u], w) : 0ull;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (r0 + 256 * u < rel1) ral_pq_store(col.data, pg.row_start + r0 + 256 * u, w, x[u]);
        }
        return;
    }
    if (!pg.optional) {
        if (P.plain_every == 0 || (item - P.item_lo) % P.plain_every) ral_pq_plain_rows(pg, col, rel0, rel1, threadIdx.x);
        return;
    }
    // PLAIN values, or a dictionary's entries through the present rows' indices
    // the page's values, or its rows' places in the indices: where its levels did not read, the items' first
    // values are not their ranks in the page
    const int64_t nvals = pg.dict_count > 0 ? (int64_t)pg.rows : (pg.data_bytes - lo) / w;
    const uint8_t* const dict = (const uint8_t*)pg.dict;
    const uint32_t* const ix = P.idx + pg.idx0;
    // this item's validity words, page-relative (rows of the next page masked off)
    ral_u32 X = 0;
    {
        const int r0 = rel0 + 32 * (int)threadIdx.x;
        if (r0 < rel1) {
            const int64_t g = pg.row_start + r0;
            const int sh = (int)(g & 31);
            const int nb = min(32, rel1 - r0);
            const ral_u32* vw = col.valid + (g >> 5);
            X = vw[0] >> sh;
            if (sh && nb > 32 - sh) X |= vw[1] << (32 - sh);
            if (nb < 32) X &= (1u << nb) - 1u;
        }
    }
    // exclusive scan of the words' popcounts
    const ral_u32 c = __popc(X);
    ral_u32 incl = c;
    for (int d = 1; d < 32; d <<= 1) {
        const ral_u32 y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_wsum[warp] = incl;
    s_word[threadIdx.x] = X;
    __syncthreads();
    ral_u32 before = 0;
    for (int k = 0; k < warp; ++k) before += s_wsum[k];
    s_base[threadIdx.x] = before + incl - c;
    __syncthreads();
    const int64_t base = (int64_t)P.item_base[item];
    // each warp takes four words (of 32 rows) per step, their loads in flight together
    for (int t0 = warp; t0 * 32 < rel1 - rel0; t0 += 32) {
        int64_t vi[4];  // the row's value, or -1
        unsigned long long x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = t0 + 8 * u, r = rel0 + 32 * t + lane;
            const ral_u32 Xw = r < rel1 ? s_word[t] : 0u;
            vi[u] = (Xw >> lane) & 1u ? base + s_base[t] + __popc(Xw & ((1u << lane) - 1u)) : -1;
        }
        if (pg.dict_count > 0) {
            uint32_t k[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = vi[u] >= 0 && vi[u] < nvals ? ix[vi[u]] : 0xffffffffu;
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = k[u] < (uint32_t)pg.dict_count ? ral_pq_value(dict, k[u], w) : 0ull;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = vi[u] >= 0 && vi[u] < nvals ? ral_pq_value(vals, vi[u], w) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = rel0 + 32 * (t0 + 8 * u) + lane;
            if (r < rel1) ral_pq_store(col.data, pg.row_start + r, w, x[u]);
        }
    }
}

// A dictionary-encoded page: after the bit width byte, the present rows' indices in
// the RLE / bit-packed hybrid (a run header varint h: h odd -> (h >> 1) groups of 8 values of the
// bit width, packed from the low bits; h even -> h >> 1 repeats of the next ceil(width / 8) bytes).
// A batch is a window of the stream: the block copies it into shared memory with 16-byte loads, thread 0
// walks the run headers in it into segments (an RLE run, or the groups of a bit-packed run that lie in
// the window), then the block writes the batch's indices from there, each checked against the
// dictionary's size.  Several blocks share a page's batches; a window inside one long run has no header,
// and only the block that writes its indices reads it.  Bound: the walk where runs are short, one chain of
// dependent instructions, in 32 bits and with a header's bytes read together (700,001 rows of three
// columns, the whole scan, against a walk byte by byte in global memory: runs of 504 values 325 -> 245 us, runs
// of 1 to 320 values 759 -> 501 us, one run a page 132 -> 125 us).

constexpr int kDictStage = 32768;  // packed index bytes staged per batch
constexpr int kDictThreads = 1024;
// Blocks of a page: each walks the run headers, block y writes batches y, y + kDictSlices, ... (24 pages of
// 131,072 indices of 6 to 12 bits, 3 to 6 batches each: 50 us with one block a page, 20 with eight).
constexpr int kDictSlices = 8;

__global__ void __launch_bounds__(kDictThreads) parquet_dict_index_kernel(const __grid_constant__ ParquetDecodeParams P) {
    __shared__ __align__(16) uint8_t s_buf[kDictStage + 64];
    __shared__ int s_row[kPqRuns + 1];
    __shared__ ral_u32 s_info[kPqRuns];  // bit-packed: the segment's first byte in s_buf; RLE: the value
    __shared__ unsigned char s_kind[kPqRuns];
    __shared__ int s_n, s_bad, s_done;
    __shared__ long long s_pos, s_rem;  // the stream offset reached, and the groups left of the run it is in
    if ((int)blockIdx.x >= P.page_hi - P.page_lo) {
        ral_pq_plain_block(P, ((int)blockIdx.x - (P.page_hi - P.page_lo)) * kDictSlices + (int)blockIdx.y);
        return;
    }
    const int p = P.page_lo + (int)blockIdx.x;
    const ParquetPage pg = P.pages[p];
    if (pg.dict_count <= 0 || pg.rows <= 0) return;
    const int n_idx = pg.optional ? (int)min((unsigned)pg.rows, P.page_present[p]) : pg.rows;
    const uint8_t* const sv = (const uint8_t*)pg.data + pg.values_off;
    const long long sbytes = (long long)pg.data_bytes - pg.values_off;
    uint32_t* const ix = P.idx + pg.idx0;
    if (n_idx <= 0) return;
    if (sbytes < 1 || sv[0] > 32) {
        if (threadIdx.x == 0 && blockIdx.y == 0) atomicAdd(P.status, 1ull);
        return;
    }
    const int bw = sv[0];
    const int vbytes = (bw + 7) >> 3;
    const uint8_t* const st = sv + 1;
    const long long nb = sbytes - 1;
    const unsigned long long mask = bw == 32 ? 0xffffffffull : ((1ull << bw) - 1ull);
    if (threadIdx.x == 0) {
        s_pos = 0;
        s_row[0] = 0;
        s_bad = 0;
        s_done = 0;
        s_rem = 0;
    }
    __syncthreads();
    bool out_of_range = false;
    for (int batch = 0;; ++batch) {
        const bool mine = batch % kDictSlices == (int)blockIdx.y;
        // the window: stream bytes [w0, w1), staged from the aligned address at or before them (inside the
        // page's buffer, which is 16-byte padded)
        const long long w0 = s_pos, w1 = min(w0 + kDictStage - 32, nb);
        const uintptr_t a0 = (uintptr_t)(st + w0) & ~(uintptr_t)15;
        const long long sbase = (long long)(a0 - (uintptr_t)st);  // stream offset of s_buf[0] (may be negative)
        if (mine || s_rem * bw <= w1 - w0) {
            const int nv = (int)(((uintptr_t)(st + w1) + 15 - a0) >> 4);
            for (int i = threadIdx.x; i < nv; i += blockDim.x)
                reinterpret_cast<uint4*>(s_buf)[i] = reinterpret_cast<const uint4*>(a0)[i];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // positions are offsets in s_buf
            const int at0 = (int)(w0 - sbase), end = (int)(w1 - sbase);
            const long long end_nb = nb - sbase;
            int k = 0, row = s_row[0], pos = at0;
            long long rem = s_rem;
            while (k < kPqRuns && row < n_idx) {
                if (rem > 0) {
                    // the groups of the bit-packed run in progress that lie in the window
                    const long long g = rem * bw <= end - pos ? rem : (end - pos) / bw;
                    if (g <= 0) break;
                    s_kind[k] = 1;
                    s_info[k] = (ral_u32)pos;
                    s_row[k++] = row;
                    row = (int)min(row + g * 8, (long long)n_idx);
                    pos += (int)g * bw;
                    rem -= g;
                    continue;
                }
                if (pos + 10 > end && w1 < nb) break;  // a header and an RLE run's value: up to ten bytes
                // eight bytes from here on: a header of one or two, and a value, are read from them
                const ral_u32* const w = reinterpret_cast<const ral_u32*>(s_buf) + (pos >> 2);
                const ral_u32 a = w[0], b = w[1], c = w[2], sh = 8u * (ral_u32)(pos & 3);
                const unsigned long long x = (unsigned long long)__funnelshift_r(b, c, sh) << 32 | __funnelshift_r(a, b, sh);
                unsigned long long h;
                ral_u32 v;  // the bytes after the header
                int hb;
                if (!(x & 0x80)) {
                    hb = 1;
                    h = x & 0x7f;
                    v = (ral_u32)(x >> 8);
                } else if (!(x & 0x8000)) {
                    hb = 2;
                    h = (x & 0x7f) | (x >> 1 & 0x3f80);
                    v = (ral_u32)(x >> 16);
                } else {
                    bool more = true;
                    h = 0;
                    for (hb = 0; hb < 6 && pos + hb < end && more; ++hb) {
                        const unsigned long long y = s_buf[pos + hb];
                        h |= (y & 0x7f) << (7 * hb);
                        more = (y & 0x80) != 0;
                    }
                    v = 0;
                    for (int j = 0; j < 4; ++j) v |= (ral_u32)s_buf[pos + hb + j] << (8 * j);
                    if (more) hb = 1 << 20;  // no header
                }
                pos += hb;
                const long long after = end_nb - pos;
                if (h & 1) rem = (long long)(h >> 1);
                if (after < 0 || ((h & 1) ? rem * bw : (long long)vbytes) > after) {
                    s_bad = 1;
                    break;
                }
                if (h & 1) continue;
                pos += vbytes;
                const int len = (int)min((long long)(h >> 1), (long long)(n_idx - row));
                if (len <= 0) continue;
                s_kind[k] = 0;
                s_info[k] = v & (ral_u32)mask;
                s_row[k++] = row;
                row += len;
            }
            s_pos = sbase + pos;
            s_rem = rem;
            s_n = k;
            s_row[k] = row;
            if (row >= n_idx) s_done = 1;
            else if (pos == at0 && k == 0) s_bad = 1;
        }
        __syncthreads();
        if (s_bad) break;
        const int n = s_n, r_lo = s_row[0], r_hi = s_row[n];
        if (!mine) {
            __syncthreads();
            if (s_done) break;
            if (threadIdx.x == 0) s_row[0] = r_hi;
            __syncthreads();
            continue;
        }
        for (int i = r_lo + (int)threadIdx.x; i < r_hi; i += kDictThreads) {
            int a = 0, b = n - 1;  // the last segment starting at or before i
            while (a < b) {
                const int m = (a + b + 1) >> 1;
                if (s_row[m] <= i) a = m;
                else b = m - 1;
            }
            ral_u32 v;
            if (s_kind[a]) {
                const int bo = (i - s_row[a]) * bw;
                const int q = (int)s_info[a] + (bo >> 3);
                const ral_u32* const w = reinterpret_cast<const ral_u32*>(s_buf) + (q >> 2);
                // up to 32 bits from bit sh of three words
                const int sh = 8 * (q & 3) + (bo & 7);  // below 32
                const unsigned long long x = (unsigned long long)w[1] << 32 | w[0];
                v = (ral_u32)(x >> sh) & (ral_u32)mask;
            } else {
                v = s_info[a];
            }
            if (v >= (ral_u32)pg.dict_count) {
                out_of_range = true;
                v = 0;
            }
            ix[i] = v;
        }
        __syncthreads();
        if (s_done) break;
        if (threadIdx.x == 0) s_row[0] = r_hi;
        __syncthreads();
    }
    // a malformed run is found by every block of the page, an index out of range by one
    const bool any = __syncthreads_or(out_of_range);
    if (threadIdx.x == 0 && (any || (s_bad && blockIdx.y == 0))) atomicAdd(P.status, 1ull);
}

cudaError_t launch_parquet_dict_indices(const ParquetDecodeParams& p, cudaStream_t st) {
    if (p.page_hi <= p.page_lo) return cudaSuccess;
    const int items = p.plain_every > 1 ? (p.item_hi - p.item_lo + p.plain_every - 1) / p.plain_every : 0;
    parquet_dict_index_kernel<<<dim3(p.page_hi - p.page_lo + (items + 4 * kDictSlices - 1) / (4 * kDictSlices), kDictSlices),
                                kDictThreads, 0, st>>>(p);
    note_launch();
    return cudaGetLastError();
}

// ---- Snappy --------------------------------------------------------------------------------
// The raw Snappy format (google/snappy format_description.txt): a varint of the uncompressed
// length, then elements, each a tag byte whose low two bits give its kind: 0 a literal (length - 1
// in the tag's upper six bits, or for 60 .. 63 in the next 1 .. 4 bytes, little-endian), followed by
// its bytes; 1 a copy of 4 + ((tag >> 2) & 7) bytes from offset ((tag >> 5) << 8 | next byte);
// 2 and 3 a copy of 1 + (tag >> 2) bytes from a 2- or 4-byte little-endian offset.  A copy reads
// the output `offset` bytes back and may overlap itself (byte i reads byte i - offset).
// One warp per page: every lane decodes the same tags from a window of the input staged in shared
// memory (so control flow stays uniform), and the lanes move an element's bytes together: byte i of
// a copy is output[op - offset + i % offset], which precedes op, so one pass suffices.

constexpr int kSnapWin = 2048;

__global__ void __launch_bounds__(256) snappy_decompress_kernel(const SnappyJob* __restrict__ jobs, int32_t n_jobs,
                                                                unsigned long long* status) {
    __shared__ uint8_t s_win[8][kSnapWin];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = (int)blockIdx.x * 8 + warp;
    if (j >= n_jobs) return;
    const SnappyJob job = jobs[j];
    uint8_t* const win = s_win[warp];
    for (int i = lane; i < job.prefix; i += 32) job.dst[i] = job.src[i - job.prefix];
    uint8_t* const out = job.dst + job.prefix;
    const uint8_t* const in = job.src;
    const int nin = job.src_bytes, nout = job.dst_bytes;
    int wbase = 0;
    auto load = [&](int at) {
        __syncwarp();
        for (int i = lane; i < kSnapWin; i += 32) win[i] = at + i < nin ? in[at + i] : 0;
        __syncwarp();
        wbase = at;
    };
    auto inb = [&](int q) -> unsigned {
        return (q >= wbase && q < wbase + kSnapWin) ? (unsigned)win[q - wbase] : (q < nin ? (unsigned)in[q] : 0u);
    };
    load(0);
    bool bad = false;
    int ip = 0, op = 0;
    {
        unsigned long long ulen = 0;
        int shift = 0;
        while (true) {
            if (ip >= nin || shift > 35) {
                bad = true;
                break;
            }
            const unsigned b = inb(ip++);
            ulen |= (unsigned long long)(b & 0x7f) << shift;
            shift += 7;
            if (!(b & 0x80)) break;
        }
        if (ulen != (unsigned long long)nout) bad = true;
    }
    while (!bad && ip < nin) {
        if (ip + 5 > wbase + kSnapWin) load(ip);  // the tag and its extra bytes in the window
        const unsigned tag = inb(ip);
        int len = 0, off = 0;
        const unsigned kind = tag & 3u;
        if (kind == 0u) {
            const unsigned l = tag >> 2;
            if (l < 60u) {
                len = (int)l + 1;
                ip += 1;
            } else {
                const int nb = (int)l - 59;
                unsigned long long v = 0;
                for (int k = 0; k < nb; ++k) v |= (unsigned long long)inb(ip + 1 + k) << (8 * k);
                if (ip + 1 + nb > nin || v >= 0x7fffffffull) {
                    bad = true;
                    break;
                }
                len = (int)v + 1;
                ip += 1 + nb;
            }
            if (len > nin - ip || len > nout - op) {
                bad = true;
                break;
            }
            for (int i = lane; i < len; i += 32) out[op + i] = (uint8_t)inb(ip + i);
            ip += len;
        } else {
            if (kind == 1u) {
                len = 4 + (int)((tag >> 2) & 7u);
                off = (int)(((tag >> 5) << 8) | inb(ip + 1));
                ip += 2;
            } else if (kind == 2u) {
                len = 1 + (int)(tag >> 2);
                off = (int)(inb(ip + 1) | inb(ip + 2) << 8);
                ip += 3;
            } else {
                len = 1 + (int)(tag >> 2);
                const unsigned long long o = (unsigned long long)inb(ip + 1) | (unsigned long long)inb(ip + 2) << 8 |
                                             (unsigned long long)inb(ip + 3) << 16 | (unsigned long long)inb(ip + 4) << 24;
                if (o > 0x7fffffffull) {
                    bad = true;
                    break;
                }
                off = (int)o;
                ip += 5;
            }
            if (ip > nin || off == 0 || off > op || len > nout - op) {
                bad = true;
                break;
            }
            __syncwarp();  // the bytes it reads, written by any lane, are visible
            for (int i = lane; i < len; i += 32) out[op + i] = out[op - off + i % off];
        }
        op += len;
        __syncwarp();
    }
    if (op != nout) bad = true;
    if (bad && lane == 0) atomicAdd(status, 1ull);
}

cudaError_t launch_snappy_decompress(const SnappyJob* jobs, int32_t n_jobs, unsigned long long* status, cudaStream_t st) {
    if (n_jobs <= 0) return cudaSuccess;
    snappy_decompress_kernel<<<(n_jobs + 7) / 8, 256, 0, st>>>(jobs, n_jobs, status);
    note_launch();
    return cudaGetLastError();
}

__global__ void parquet_level_lengths_kernel(const __grid_constant__ ParquetDecodeParams P) {
    const int p = P.page_lo + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (p >= P.page_hi) return;
    ParquetPage& pg = P.pages[p];
    if (pg.levels >= 0) return;
    const uint8_t* const d = (const uint8_t*)pg.data;
    long long lev = -1;
    if (pg.data_bytes >= 4) lev = (long long)((unsigned)d[0] | (unsigned)d[1] << 8 | (unsigned)d[2] << 16 | (unsigned)d[3] << 24);
    if (lev < 0 || 4 + lev > pg.data_bytes) {
        atomicAdd(P.status, 1ull);
        pg.levels = 0;  // the later kernels then find nothing to read
        pg.values_off = pg.data_bytes;
    } else {
        pg.levels = (int32_t)lev;
        pg.values_off = 4 + (int32_t)lev;
    }
}

cudaError_t launch_parquet_level_lengths(const ParquetDecodeParams& p, cudaStream_t st) {
    if (p.page_hi <= p.page_lo) return cudaSuccess;
    parquet_level_lengths_kernel<<<(p.page_hi - p.page_lo + 255) / 256, 256, 0, st>>>(p);
    note_launch();
    return cudaGetLastError();
}

// One copy by threads t, t + step, ...: 16-byte words where source and destination agree in alignment.
__device__ __forceinline__ void ral_copy(const CopyJob& j, int64_t t, int64_t step) {
    const uintptr_t s = (uintptr_t)j.src, d = (uintptr_t)j.dst;
    if (((s ^ d) & 15) == 0) {
        const int64_t lead = (int64_t)((16 - (s & 15)) & 15);
        const int64_t head = j.bytes < lead ? j.bytes : lead;
        for (int64_t i = t; i < head; i += step) j.dst[i] = j.src[i];
        const int64_t nv = (j.bytes - head) >> 4;
        const uint4* sv = reinterpret_cast<const uint4*>(j.src + head);
        uint4* dv = reinterpret_cast<uint4*>(j.dst + head);
        for (int64_t i = t; i < nv; i += step) dv[i] = sv[i];
        for (int64_t i = head + nv * 16 + t; i < j.bytes; i += step) j.dst[i] = j.src[i];
    } else if (((s ^ d) & 3) == 0) {
        const int64_t lead = (int64_t)((4 - (s & 3)) & 3);
        const int64_t head = j.bytes < lead ? j.bytes : lead;
        for (int64_t i = t; i < head; i += step) j.dst[i] = j.src[i];
        const int64_t nv = (j.bytes - head) >> 2;
        const ral_u32* sv = reinterpret_cast<const ral_u32*>(j.src + head);
        ral_u32* dv = reinterpret_cast<ral_u32*>(j.dst + head);
        for (int64_t i = t; i < nv; i += step) dv[i] = sv[i];
        for (int64_t i = head + nv * 4 + t; i < j.bytes; i += step) j.dst[i] = j.src[i];
    } else {
        for (int64_t i = t; i < j.bytes; i += step) j.dst[i] = j.src[i];
    }
}

__device__ __forceinline__ void ral_fill(const CopyJob& j, ral_u32 byte, int64_t t, int64_t step) {
    const uintptr_t d = (uintptr_t)j.dst;
    const int64_t lead = (int64_t)((16 - (d & 15)) & 15);
    const int64_t head = j.bytes < lead ? j.bytes : lead;
    const ral_u32 w = byte * 0x01010101u;
    for (int64_t i = t; i < head; i += step) j.dst[i] = (uint8_t)byte;
    const int64_t nv = (j.bytes - head) >> 4;
    uint4* dv = reinterpret_cast<uint4*>(j.dst + head);
    for (int64_t i = t; i < nv; i += step) dv[i] = make_uint4(w, w, w, w);
    for (int64_t i = head + nv * 16 + t; i < j.bytes; i += step) j.dst[i] = (uint8_t)byte;
}

// One block per job.  In place of a memset for each mask part and counter and a copy for each dictionary:
// sixteen calls of a four-column scan, 1.5 to 3 us each.
__global__ void __launch_bounds__(256) prepare_jobs_kernel(const PrepareJob* __restrict__ jobs) {
    const PrepareJob j = jobs[blockIdx.x];
    if (j.copy.src) ral_copy(j.copy, threadIdx.x, blockDim.x);
    else ral_fill(j.copy, (ral_u32)j.fill & 0xffu, threadIdx.x, blockDim.x);
}

__global__ void __launch_bounds__(256) copy_list_kernel(const __grid_constant__ CopyList list) {
    ral_copy(list.job[blockIdx.y], (int64_t)blockIdx.x * 256 + threadIdx.x, (int64_t)gridDim.x * 256);
}

cudaError_t launch_copy_list(const CopyList& list, cudaStream_t st) {
    int64_t most = 0;
    for (int k = 0; k < list.n; k++) most = std::max(most, list.job[k].bytes);
    if (most <= 0) return cudaSuccess;
    // 4 of the 16-byte words a thread, up to the device's threads for all jobs together
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((most + 16383) / 16384, ((int64_t)device_sms() * 8 + list.n - 1) / list.n));
    copy_list_kernel<<<dim3((unsigned)blocks, (unsigned)list.n), 256, 0, st>>>(list);
    note_launch();
    return cudaGetLastError();
}

__global__ void __launch_bounds__(96) copy_headers_kernel(const HeaderJob* __restrict__ jobs, unsigned long long* __restrict__ dst) {
    const HeaderJob j = jobs[blockIdx.x];
    if ((int64_t)threadIdx.x < j.words) dst[(size_t)blockIdx.x * 67 + threadIdx.x] = __ldcg(j.src + threadIdx.x);
}

cudaError_t launch_copy_headers(const HeaderJob* jobs, int32_t n, unsigned long long* dst, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    copy_headers_kernel<<<n, 96, 0, st>>>(jobs, dst);
    note_launch();
    return cudaGetLastError();
}

// In place of a memset per scratch area and output mask before a filter or a text scan, some 2 us each, one
// after the other (9M rows of six columns with nulls, half of them kept: 183 -> 161 us; the masks of a 20M-line text scan 799 -> 786 us).
__global__ void __launch_bounds__(256) zero_list_kernel(const __grid_constant__ ZeroList list) {
    ral_fill(CopyJob{nullptr, (uint8_t*)list.p[blockIdx.y], 4 * list.words[blockIdx.y]}, 0u,
             (int64_t)blockIdx.x * 256 + threadIdx.x, (int64_t)gridDim.x * 256);
}

cudaError_t launch_zero_list(const ZeroList& list, cudaStream_t st) {
    if (list.n <= 0) return cudaSuccess;
    int64_t most = 0;
    for (int k = 0; k < list.n; k++) most = std::max(most, list.words[k]);
    // 4 of the 16-byte words a thread, up to the device's threads for all ranges together
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((most + 4095) / 4096, ((int64_t)device_sms() * 8 + list.n - 1) / list.n));
    zero_list_kernel<<<dim3((unsigned)blocks, (unsigned)list.n), 256, 0, st>>>(list);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_prepare_jobs(const PrepareJob* jobs, int32_t n_jobs, cudaStream_t st) {
    if (n_jobs <= 0) return cudaSuccess;
    prepare_jobs_kernel<<<n_jobs, 256, 0, st>>>(jobs);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_parquet_levels(const ParquetDecodeParams& p, cudaStream_t st) {
    if (p.page_hi <= p.page_lo) return cudaSuccess;
    parquet_levels_kernel<<<p.page_hi - p.page_lo + (p.item_hi - p.item_lo + 3) / 4, kLevelThreads, 0, st>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_parquet_values(const ParquetDecodeParams& p, cudaStream_t st) {
    if (p.item_hi <= p.item_lo) return cudaSuccess;
    parquet_values_kernel<<<p.item_hi - p.item_lo, 256, 0, st>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_category_remap(int32_t* codes, int64_t n, const int32_t* table, int32_t table_n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 152 * 8));
    category_remap_kernel<<<(int)blocks, threads, 0, st>>>(codes, n, table, table_n);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_category_insert(int32_t* codes, int64_t n, int32_t pos, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 152 * 8));
    category_insert_kernel<<<(int)blocks, threads, 0, st>>>(codes, n, pos);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gather_columns(const GatherColumnsParams& p, cudaStream_t st) {
    if (p.n_out <= 0 || p.num_columns <= 0) return cudaSuccess;
    int dev = 0, sms = 1, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gather_columns_kernel, 256, 0);
    if (per_sm < 1) per_sm = 1;
    const int64_t steps = (p.n_out + 32 * kGatherRowsPerLane - 1) / (32 * kGatherRowsPerLane);
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((steps + 7) / 8, (int64_t)sms * per_sm));
    gather_columns_kernel<<<(int)grid, 256, 0, st>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gather_probe(const GatherColumnsParams& p, int32_t* scattered, cudaStream_t st) {
    static_assert(kGatherProbeRows >= 32 * kGatherSamples, "a sample starts within the index");
    gather_probe_kernel<<<1, 256, 0, st>>>(p, scattered);
    note_launch();
    return cudaGetLastError();
}

}  // namespace ral
