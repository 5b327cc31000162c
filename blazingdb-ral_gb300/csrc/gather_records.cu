// gather_records.cu — a scattered gather of several columns by way of row records.
//
// A random element costs a DRAM access whatever its width: six columns of 100M rows by a permutation read
// over 500 bytes per row for 29 bytes of elements.  Here the columns are first laid out as records (a
// row's elements back to back, then one validity bit per masked column, padded to 16, 32 or 64 bytes), a
// streaming pass; a row of the gather then costs one random access for all of its columns.
//
// Six columns of 100M rows (29 bytes and six validity bits a row) by a permutation: 13.6 ms straight from
// the columns, 3.72 ms here; 30M rows 3.16 / 1.16, 4M rows 0.236 / 0.180, 1M rows 0.083 / 0.072 ms (below
// that the two extra launches cost more than the accesses saved).  Of 30M rows' 1.16 ms the pack takes
// 0.33 (60 bytes a row streamed) and the gather 0.70: 43 G random records a second, a rate that the card
// does not exceed for 8-byte or 32-byte accesses, 64 or 128 bytes fetched, alike.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_rt.cuh"
#include "engine.h"
#include "kernels.h"

namespace ral {

namespace {

constexpr int kThreads = 256;
constexpr int kRecordColumns = 64;

struct RecordColumn {
    const void* in;
    const uint32_t* in_valid;
    void* out;
    uint32_t* out_valid;
    unsigned long long* count;
    int32_t width, at;    // the element's place in the record
    int32_t bit;          // its validity bit's place in the record's bits, or -1: always valid
    int32_t pad;
};
struct RecordParams {
    RecordColumn col[kRecordColumns];
    const void* idx;
    const int32_t* scattered;  // 0: nothing to do here
    uint4* records;
    int64_t n_in, n_out;
    int32_t num_columns, idx_width;
    int32_t bits_at;           // the byte where the validity bits start
    int32_t bits_bytes;        // their bytes
};

// A warp's step: kRows rows a lane (row 32 k + lane), whose records pass through shared memory between
// the columns (a row a lane) and the records (16 bytes a lane, consecutive lanes on consecutive bytes).
// A record takes an odd number of words there, so both sides spread over the banks.
template <int W>
struct Step {
    static constexpr int kRows = W == 16 ? 2 : 4;
    static constexpr int kStride = W + 1;
    static constexpr int kParts = W / 4;             // 16-byte parts of a record
    static constexpr int kMoves = kRows * kParts;    // of 32 parts each
};

// One column's elements of a step into the records: all loads, then the stores to shared memory.
template <int W, typename E>
__device__ __forceinline__ void pack_column(const RecordColumn& col, ral_i64 base, int left, int lane, ral_u32* rec,
                                            ral_u32 (&bits)[Step<W>::kRows][2]) {
    using S = Step<W>;
    const E* const in = (const E*)col.in + base;
    E v[S::kRows];
    ral_u32 m[S::kRows];
#pragma unroll
    for (int k = 0; k < S::kRows; ++k) {
        const int i = 32 * k + lane;
        v[k] = i < left ? __ldcs(in + i) : E(0);
        m[k] = col.bit >= 0 && 32 * k < left ? __ldg(col.in_valid + (base >> 5) + k) : 0u;  // one word for the warp's 32 rows
    }
    ral_u32* const at = rec + lane * S::kStride + (col.at >> 2);
#pragma unroll
    for (int k = 0; k < S::kRows; ++k) {
        ral_u32* const q = at + 32 * k * S::kStride;
        if constexpr (sizeof(E) == 8) {
            q[0] = (ral_u32)(unsigned long long)v[k];
            q[1] = (ral_u32)((unsigned long long)v[k] >> 32);
        } else {
            *(E*)((char*)q + (col.at & 3)) = v[k];
        }
    }
    if (col.bit >= 0) {
        const int b = col.bit & 31;
#pragma unroll
        for (int k = 0; k < S::kRows; ++k) {
            const ral_u32 bit = ((m[k] >> lane) & 1u) << b;
            if (col.bit < 32) bits[k][0] |= bit;
            else bits[k][1] |= bit;
        }
    }
}

// Records of W words: bound by the streams (the columns read once, the records written).  Four blocks an
// SM: at six the compiler has too few registers to keep a column's loads together (100M rows of six
// columns: 4.24 ms in all against 3.72).
template <int W>
__global__ void __launch_bounds__(kThreads, 4) record_pack_kernel(const __grid_constant__ RecordParams P) {
    if (*P.scattered == 0) return;
    using S = Step<W>;
    __shared__ ral_u32 s_rec[kThreads / 32][32 * S::kRows * S::kStride];
    ral_u32* const rec = s_rec[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const ral_i64 gwarp = ((ral_i64)blockIdx.x * kThreads + threadIdx.x) >> 5, nwarp = ((ral_i64)gridDim.x * kThreads) >> 5;
    constexpr ral_i64 rows = 32 * S::kRows;
    for (ral_i64 base = gwarp * rows; base < P.n_in; base += nwarp * rows) {
        const int left = (int)min(P.n_in - base, rows);
        ral_u32 bits[S::kRows][2];  // the validity bits, up to 64 columns'
#pragma unroll
        for (int k = 0; k < S::kRows; ++k) bits[k][0] = bits[k][1] = 0u;
        __syncwarp();
        for (int c = 0; c < P.num_columns; ++c) {
            const RecordColumn& col = P.col[c];
            switch (col.width) {
            case 8: pack_column<W, long long>(col, base, left, lane, rec, bits); break;
            case 4: pack_column<W, int>(col, base, left, lane, rec, bits); break;
            case 2: pack_column<W, short>(col, base, left, lane, rec, bits); break;
            default: pack_column<W, signed char>(col, base, left, lane, rec, bits); break;
            }
        }
        // the bits, a byte at a time
        for (int b = 0; b < P.bits_bytes; ++b)
#pragma unroll
            for (int k = 0; k < S::kRows; ++k)
                ((unsigned char*)(rec + (32 * k + lane) * S::kStride))[P.bits_at + b] =
                    (unsigned char)((b < 4 ? bits[k][0] : bits[k][1]) >> (8 * (b & 3)));
        __syncwarp();
        uint4* const out = P.records + base * S::kParts;
#pragma unroll
        for (int t = 0; t < S::kMoves; ++t) {
            const int part = 32 * t + lane, row = part / S::kParts;
            const ral_u32* const q = rec + row * S::kStride + 4 * (part % S::kParts);
            if (row < left) out[part] = make_uint4(q[0], q[1], q[2], q[3]);
        }
    }
}

__device__ __forceinline__ ral_i64 index_at(const RecordParams& P, ral_i64 i) {
    switch (P.idx_width) {
    case 1: return (ral_i64)__ldcs((const signed char*)P.idx + i);
    case 2: return (ral_i64)__ldcs((const short*)P.idx + i);
    case 4: return (ral_i64)__ldcs((const int*)P.idx + i);
    default: return (ral_i64)__ldcs((const long long*)P.idx + i);
    }
}

// One column's elements of a step from the records; returns its valid rows.
template <int W, typename E>
__device__ __forceinline__ ral_u32 unpack_column(const RecordParams& P, const RecordColumn& col, ral_i64 base, int left, int lane,
                                                 const ral_u32* rec, const bool (&ok)[Step<W>::kRows]) {
    using S = Step<W>;
    E* const out = (E*)col.out + base;
    const ral_u32* const at = rec + lane * S::kStride + (col.at >> 2);
#pragma unroll
    for (int k = 0; k < S::kRows; ++k) {
        const ral_u32* const q = at + 32 * k * S::kStride;
        E v;
        if constexpr (sizeof(E) == 8) v = (E)((unsigned long long)q[1] << 32 | q[0]);
        else v = *(const E*)((const char*)q + (col.at & 3));
        if (ok[k]) __stcs(out + 32 * k + lane, v);
    }
    ral_u32 cnt = 0;
    if (col.out_valid) {
        const int b = 8 * P.bits_at + (col.bit >= 0 ? col.bit : 0);
        const ral_u32* const mq = rec + lane * S::kStride + (b >> 5);
#pragma unroll
        for (int k = 0; k < S::kRows; ++k) {
            const ral_u32 m = col.bit >= 0 ? mq[32 * k * S::kStride] >> (b & 31) : 1u;
            const ral_u32 word = __ballot_sync(0xffffffffu, ok[k] && (m & 1u));
            if (lane == k && 32 * k < left) col.out_valid[(base >> 5) + k] = word;
            cnt += __popc(word);
        }
    }
    return cnt;
}

// 16 bytes of a record.  The record's 64-byte DRAM access is all that is wanted: without the qualifier a
// miss fetches the 128 bytes around it (30M random 32-byte records read 3.7 GB in 737 us; 2.0 GB in 695 with it).
__device__ __forceinline__ uint4 load_part(const uint4* p) {
    uint4 v;
    asm("ld.global.L2::64B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// A record is read by kParts neighbouring lanes with one instruction, so that it is one access; a
// column's 32 elements leave as one contiguous store.  Bound by the random accesses.  Three blocks an SM
// (four: 3.92 ms against 3.72) and 128 rows a step (256, with half the blocks: 5.68 ms).
template <int W>
__global__ void __launch_bounds__(kThreads, 3) record_gather_kernel(const __grid_constant__ RecordParams P) {
    if (*P.scattered == 0) return;
    using S = Step<W>;
    __shared__ ral_u32 s_rec[kThreads / 32][32 * S::kRows * S::kStride];
    __shared__ ral_u32 s_cnt[kRecordColumns];
    if (threadIdx.x < kRecordColumns) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    ral_u32* const rec = s_rec[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const ral_i64 gwarp = ((ral_i64)blockIdx.x * kThreads + threadIdx.x) >> 5, nwarp = ((ral_i64)gridDim.x * kThreads) >> 5;
    constexpr ral_i64 rows = 32 * S::kRows;
    auto indices = [&](ral_i64 base, ral_i64 (&j)[S::kRows]) {
#pragma unroll
        for (int k = 0; k < S::kRows; ++k) j[k] = base + 32 * k + lane < P.n_out ? index_at(P, base + 32 * k + lane) : -1;
    };
    ral_i64 next[S::kRows];  // a step's indices are read a step ahead
    indices(gwarp * rows, next);
    for (ral_i64 base = gwarp * rows; base < P.n_out; base += nwarp * rows) {
        const int left = (int)min(P.n_out - base, rows);
        ral_i64 j[S::kRows];
        bool ok[S::kRows];
#pragma unroll
        for (int k = 0; k < S::kRows; ++k) {
            ok[k] = next[k] >= 0 && next[k] < P.n_in;
            j[k] = ok[k] ? next[k] : 0;
        }
        indices(base + nwarp * rows, next);
        uint4 v[S::kMoves];
#pragma unroll
        for (int t = 0; t < S::kMoves; ++t) {
            const int part = 32 * t + lane, row = part / S::kParts;
            const ral_i64 x = __shfl_sync(0xffffffffu, j[t / S::kParts], row & 31);
            v[t] = load_part(P.records + x * S::kParts + part % S::kParts);
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < S::kMoves; ++t) {
            const int part = 32 * t + lane, row = part / S::kParts;
            ral_u32* const q = rec + row * S::kStride + 4 * (part % S::kParts);
            q[0] = v[t].x;
            q[1] = v[t].y;
            q[2] = v[t].z;
            q[3] = v[t].w;
        }
        __syncwarp();
        for (int c = 0; c < P.num_columns; ++c) {
            const RecordColumn& col = P.col[c];
            ral_u32 cnt;
            switch (col.width) {
            case 8: cnt = unpack_column<W, long long>(P, col, base, left, lane, rec, ok); break;
            case 4: cnt = unpack_column<W, int>(P, col, base, left, lane, rec, ok); break;
            case 2: cnt = unpack_column<W, short>(P, col, base, left, lane, rec, ok); break;
            default: cnt = unpack_column<W, signed char>(P, col, base, left, lane, rec, ok); break;
            }
            if (lane == 0 && cnt) atomicAdd(&s_cnt[c], cnt);
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < P.num_columns && s_cnt[threadIdx.x] && P.col[threadIdx.x].count)
        atomicAdd(P.col[threadIdx.x].count, (unsigned long long)s_cnt[threadIdx.x]);
}

// A group's columns (of which some may follow in p): their places in the record.
void place_group(const GatherColumnsParams& p, const GatherGroup& group, RecordParams& P) {
    // widest first, so that every element is aligned; the bits after the last
    int at = 0, bit = 0;
    P.num_columns = 0;
    for (int w = 8; w >= 1; w /= 2)
        for (int c = group.from; c < group.to; c++) {
            const GatherColumn& g = p.col[c];
            if (g.width != w) continue;
            RecordColumn& r = P.col[P.num_columns++];
            r.in = g.in;
            r.in_valid = g.in_valid;
            r.out = g.out;
            r.out_valid = g.out_valid;
            r.count = p.valid_counts && g.out_valid ? p.valid_counts + c : nullptr;
            r.width = w;
            r.at = at;
            r.bit = g.in_valid && g.out_valid ? bit++ : -1;
            at += w;
        }
    P.bits_at = at;
    P.bits_bytes = (bit + 7) / 8;
}

template <int W>
void group_passes(const RecordParams& P, int grid, cudaStream_t st) {
    record_pack_kernel<W><<<grid, kThreads, 0, st>>>(P);
    record_gather_kernel<W><<<grid, kThreads, 0, st>>>(P);
    note_launch();
    note_launch();
}

}  // namespace

// Columns are taken in order, as many as fit a record; the record is then the smallest that holds them.  Records of
// 64 bytes are the fewest passes; where the input's rows make that more than `most` bytes, 32 or 16.
int gather_groups(const GatherColumnsParams& p, int64_t most, GatherGroup* groups, int64_t* bytes) {
    *bytes = 0;
    int64_t width = 64;
    while (width >= 16 && p.n_in * width > most) width /= 2;
    int n = 0;
    for (int from = 0; from < p.num_columns; n++) {
        int size = 0, elements = 0, masks = 0, to = from;
        for (; to < p.num_columns; to++) {
            const int e = elements + p.col[to].width, m = masks + (p.col[to].in_valid && p.col[to].out_valid ? 1 : 0);
            if (to > from && e + (m + 7) / 8 > width) break;
            elements = e;
            masks = m;
            size = e + (m + 7) / 8;
        }
        groups[n] = GatherGroup{from, to, size <= 16 ? 16 : size <= 32 ? 32 : 64};
        // a record of one column, or one less than half full, costs more than the accesses it saves (eight columns
        // of 8 bytes and a ninth, 8M rows: 565 us straight, 641 with it in records of its own; two of one byte 598, 631)
        if (to - from < 2 || size < 8 || groups[n].record > width) groups[n].record = 0;
        *bytes = std::max(*bytes, p.n_in * groups[n].record);
        from = to;
    }
    return n;
}

cudaError_t launch_gather_records(const GatherColumnsParams& p, const GatherGroup* groups, int n_groups, void* records, cudaStream_t st) {
    RecordParams P{};
    P.idx = p.idx;
    P.idx_width = p.idx_width;
    P.n_in = p.n_in;
    P.n_out = p.n_out;
    P.scattered = p.scattered;
    P.records = (uint4*)records;
    const int grid = (int)std::min<int64_t>((int64_t)device_sms() * 8, (std::max(p.n_in, p.n_out) + kThreads - 1) / kThreads);
    for (int g = 0; g < n_groups; g++) {
        if (!groups[g].record) continue;
        place_group(p, groups[g], P);
        if (groups[g].record == 16) group_passes<4>(P, grid, st);
        else if (groups[g].record == 32) group_passes<8>(P, grid, st);
        else group_passes<16>(P, grid, st);
        if (cudaError_t e = cudaGetLastError()) return e;
    }
    return cudaSuccess;
}

}  // namespace ral
