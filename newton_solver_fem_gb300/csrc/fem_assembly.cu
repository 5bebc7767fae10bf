// Deterministic BSR assembly of A = M + h^2 K~ + h C_s into the SELL-32 layout.
//
// The reference writes every element/constant block as a triplet and either
// sorts them (bsr_set_from_triplets) or scatters them with float atomics into
// precomputed slots (sparse_update.py:9-59).  Here the setup builds, once, the
// list of contributing triplets of every matrix slot in ascending triplet order
// (the reference layout [P | 2S | 3Tri | 16T | 64H]), and each refresh sums that list
// in order: no atomics, bit-identical results run to run.  The thread that
// owns a diagonal slot also writes that row's preconditioner block
// (kernels.py:1836-1849 fused into the assembly epilogue).
#include <algorithm>

#include "fem_internal.cuh"
#include "fem_math.cuh"

namespace fem {
namespace {

// One thread per SELL entry: sum its contributing triplet blocks in ascending
// triplet order.  Contributor places and values are loaded kGatherBatch at a time
// before any is added, so that many independent loads are in flight per thread.
// The first P triplets are the per-node constant diagonal blocks, so an entry
// is on the diagonal exactly when its first (smallest) contributor is below
// P, and that is its row: no row or column index is read.  At most 40
// registers, so 6 CTAs (48 warps) share an SM.  Reading 36 stored blocks a hex in groups of 16 hexes
// instead of 64 a hex took it from 98.6 to 73.2 us on 48^3 Hex8 (3.05 million blocks; 300 MB, 4.1 TB/s).
constexpr int kGatherBatch = 4;

__global__ void __launch_bounds__(256, 6) gather_kernel(int64_t nsell, int P, const int* __restrict__ cptr,
                              const unsigned* __restrict__ contrib,
                              const TripletPlanes trip, float4* __restrict__ valA, float4* __restrict__ valB,
                              float* __restrict__ valC, float* __restrict__ minv, int precond, int clear_empty) {
    chained_start();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nsell) return;
    const int c0 = cptr[e], c1 = cptr[e + 1];
    if (c0 == c1) {
        // padding is zero since setup; a reserved entry whose last contributor
        // left (streaming assembly) is cleared to an exact zero
        if (clear_empty) {
            valA[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            valB[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            valC[e] = 0.0f;
        }
        return;
    }
    float b[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) b[k] = 0.0f;
    unsigned first = 0;
    for (int c = c0; c < c1; c += kGatherBatch) {
        unsigned id[kGatherBatch];
#pragma unroll
        for (int u = 0; u < kGatherBatch; ++u) id[u] = c + u < c1 ? __ldg(contrib + c + u) : 0u;
        if (c == c0) first = id[0] >> 1;
        float v[kGatherBatch][9];
#pragma unroll
        for (int u = 0; u < kGatherBatch; ++u) {
            const size_t t = id[u] >> 1;
            const float4 pa = __ldg(trip.a + t), pb = __ldg(trip.b + t);
            const float pc = __ldg(trip.c + t);
            v[u][0] = pa.x; v[u][1] = pa.y; v[u][2] = pa.z; v[u][3] = pa.w;
            v[u][4] = pb.x; v[u][5] = pb.y; v[u][6] = pb.z; v[u][7] = pb.w;
            v[u][8] = pc;
        }
#pragma unroll
        for (int u = 0; u < kGatherBatch; ++u)
            if (c + u < c1) {
                const bool flip = id[u] & 1u;  // a block below its element's diagonal: the transpose of the stored one
                b[0] += v[u][0];
                b[1] += flip ? v[u][3] : v[u][1];
                b[2] += flip ? v[u][6] : v[u][2];
                b[3] += flip ? v[u][1] : v[u][3];
                b[4] += v[u][4];
                b[5] += flip ? v[u][7] : v[u][5];
                b[6] += flip ? v[u][2] : v[u][6];
                b[7] += flip ? v[u][5] : v[u][7];
                b[8] += v[u][8];
            }
    }
    valA[e] = make_float4(b[0], b[1], b[2], b[3]);
    valB[e] = make_float4(b[4], b[5], b[6], b[7]);
    valC[e] = b[8];
    if (first < (unsigned)P) {
        const unsigned row = first;
        float inv[9];
        if (precond == FEM_PRECOND_DIAG) inverse_point_diagonal(b, inv);
        else inverse_diagonal_block(b, inv);
        float* o = minv + 9 * (int64_t)row;
#pragma unroll
        for (int k = 0; k < 9; ++k) o[k] = inv[k];
    }
}

// The reference's triplets, row-major 9 floats per block, from the stored blocks.
__global__ void export_triplets_kernel(int64_t ntrip, const TripletMap map, const TripletPlanes trip,
                                       float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntrip) return;
    const unsigned p = map.place(i);
    const size_t t = p >> 1;
    const float4 a = trip.a[t], b = trip.b[t];
    float* o = out + 9 * i;
    const bool flip = p & 1u;
    o[0] = a.x;
    o[flip ? 3 : 1] = a.y;
    o[flip ? 6 : 2] = a.z;
    o[flip ? 1 : 3] = a.w;
    o[4] = b.x;
    o[flip ? 7 : 5] = b.y;
    o[flip ? 2 : 6] = b.z;
    o[flip ? 5 : 7] = b.w;
    o[8] = trip.c[t];
}

// The matrix in BSR form: the pattern, and the SELL blocks as values (rows ascending, a row's columns in
// its SELL order), 36 bytes a block.  The rows of a slice are one run of BSR values, so a CTA reads the
// slice's planes coalesced, places the blocks in that order in shared memory and writes the run with one
// bulk copy (its ends, up to a 16-byte boundary, by single stores).  3.05 million blocks take 52 us; 62
// with a warp storing each row's run of eight columns, 115 with a thread per block.  The first
// pattern_blocks CTAs copy the pattern (two device copies after the kernel took 8 us).
constexpr int kExportThreads = 128, kExportMaxWidth = 64;

struct ExportArgs {
    int pattern_blocks;
    const int* __restrict__ slice_ptr;
    const int2* __restrict__ meta;
    const unsigned* __restrict__ row_info;
    const int* __restrict__ offsets;
    const int* __restrict__ columns;
    int64_t nnzb;
    int P;
    const float4* __restrict__ valA;
    const float4* __restrict__ valB;
    const float* __restrict__ valC;
    int* __restrict__ out_offsets;
    int* __restrict__ out_columns;
    float* __restrict__ out;
};

__global__ void __launch_bounds__(kExportThreads) export_bsr_kernel(const ExportArgs a) {
    extern __shared__ __align__(16) float tile[];
    if ((int)blockIdx.x < a.pattern_blocks) {
        const int64_t i0 = (int64_t)blockIdx.x * kExportThreads + threadIdx.x;
        const int64_t step = (int64_t)a.pattern_blocks * kExportThreads;
        if (a.out_offsets != nullptr)
            for (int64_t i = i0; i <= a.P; i += step) a.out_offsets[i] = a.offsets[i];
        if (a.out_columns != nullptr)
            for (int64_t i = i0; i < a.nnzb; i += step) a.out_columns[i] = a.columns[i];
        return;
    }
    const int sl = blockIdx.x - a.pattern_blocks;
    const int lane = threadIdx.x & 31;
    const int base = a.slice_ptr[sl], width = a.slice_ptr[sl + 1] - base;
    const int2 m = a.meta[sl];
    const int run0 = a.offsets[m.x], run1 = a.offsets[m.x + m.y];
    const bool live = lane < m.y;
    const int len = live ? (int)(a.row_info[m.x + lane] & ~kFixedBit) : 0;
    float* out = a.out + 9 * (size_t)run0;
    const int shift = (int)((reinterpret_cast<uintptr_t>(out) >> 2) & 3);  // of both copies, in floats
    float* t = tile + shift;
    float* row = t + 9 * (live ? a.offsets[m.x + lane] - run0 : 0);
#pragma unroll 4
    for (int k = threadIdx.x >> 5; k < width; k += kExportThreads / 32)
        if (k < len) {
            const size_t e = (size_t)(base + k) * kSlice + lane;
            const float4 va = __ldg(a.valA + e), vb = __ldg(a.valB + e);
            float* o = row + 9 * k;
            o[0] = va.x; o[1] = va.y; o[2] = va.z; o[3] = va.w;
            o[4] = vb.x; o[5] = vb.y; o[6] = vb.z; o[7] = vb.w;
            o[8] = __ldg(a.valC + e);
        }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the placed blocks visible to the bulk copy
    __syncthreads();
    const int n = 9 * (run1 - run0), head = min(n, (4 - shift) & 3), bulk = (n - head) & ~3;
    if (threadIdx.x == 0 && bulk > 0) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out + head),
                     "r"((unsigned)__cvta_generic_to_shared(t + head)), "r"(4 * bulk)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    if ((int)threadIdx.x - 32 >= 0 && (int)threadIdx.x - 32 < head) out[threadIdx.x - 32] = t[threadIdx.x - 32];
    const int tail = head + bulk + (int)threadIdx.x - 64;
    if (threadIdx.x >= 64 && tail < n) out[tail] = t[tail];
}

// The same for slices too wide for that: a warp takes kExportColumns block columns of a slice at a time
// (blockIdx.y, and on by gridDim.y, which ends at 65,535) and writes each row's run of them (62 us for the 3.05
// million blocks).
constexpr int kExportColumns = 8, kExportWarps = 4;
constexpr int kExportRow = 9 * kExportColumns + 1;  // padded: the 32 rows of a column in distinct banks

__global__ void __launch_bounds__(32 * kExportWarps) export_columns_kernel(
    int nslices, const int* __restrict__ slice_ptr, const int2* __restrict__ meta, const unsigned* __restrict__ row_info,
    const int* __restrict__ offsets, const float4* __restrict__ valA, const float4* __restrict__ valB,
    const float* __restrict__ valC, float* __restrict__ out) {
    __shared__ float tile[kExportWarps][32 * kExportRow];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int sl = blockIdx.x * kExportWarps + w;
    if (sl >= nslices) return;  // the whole warp
    const int base = slice_ptr[sl], width = slice_ptr[sl + 1] - base;
    const int2 m = meta[sl];
    const bool live = lane < m.y;
    const int len = live ? (int)(row_info[m.x + lane] & ~kFixedBit) : 0;
    const int start = live ? offsets[m.x + lane] : 0;
    float* t = tile[w];
    for (int k0 = blockIdx.y * kExportColumns; k0 < width; k0 += gridDim.y * kExportColumns) {
#pragma unroll
        for (int u = 0; u < kExportColumns; ++u)
            if (k0 + u < len) {
                const size_t e = (size_t)(base + k0 + u) * kSlice + lane;
                const float4 a = __ldg(valA + e), b = __ldg(valB + e);
                float* o = t + lane * kExportRow + 9 * u;
                o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
                o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
                o[8] = __ldg(valC + e);
            }
        __syncwarp();
        for (int r = 0; r < m.y; ++r) {
            const int n = 9 * min(kExportColumns, __shfl_sync(0xffffffffu, len, r) - k0);
            float* o = out + 9 * ((size_t)__shfl_sync(0xffffffffu, start, r) + k0);
            for (int i = lane; i < n; i += 32) o[i] = t[r * kExportRow + i];
        }
        __syncwarp();  // the tile is read before it is written again
    }
}

}  // namespace

cudaError_t launch_gather(Handle& h, cudaStream_t s) {
    if (h.nsell == 0) return cudaSuccess;
    int threads = 256;
    int64_t blocks = (h.nsell + threads - 1) / threads;
    launch_maybe_chained(blocks <= kChainedBlocks, gather_kernel, (unsigned)blocks, threads, 0, s, h.nsell, h.P,
                         h.sell_cptr, reinterpret_cast<const unsigned*>(h.sell_contrib), h.trip, h.valA, h.valB, h.valC,
                         h.minv, h.precond, h.streaming);
    return cudaGetLastError();
}

cudaError_t launch_export_bsr(Handle& h, int* offsets, int* columns, float* values, cudaStream_t s) {
    if (h.nslices == 0) return cudaSuccess;
    const bool narrow = h.slice_width <= kExportMaxWidth;
    ExportArgs a;
    a.pattern_blocks = offsets != nullptr || columns != nullptr
                           ? std::min(1024, blocks_for(std::max<int64_t>(h.nnzb, h.P + 1), 8 * kExportThreads))
                           : 0;
    a.slice_ptr = h.slice_ptr;
    a.meta = h.slice_meta;
    a.row_info = h.row_info;
    a.offsets = h.bsr_offsets;
    a.columns = h.bsr_columns;
    a.nnzb = h.nnzb;
    a.P = h.P;
    a.valA = h.valA;
    a.valB = h.valB;
    a.valC = h.valC;
    a.out_offsets = offsets;
    a.out_columns = columns;
    a.out = values;
    const int slices = values != nullptr && narrow ? h.nslices : 0;
    const size_t bytes = slices > 0 ? (9 * (size_t)h.slice_width * kSlice + 4) * sizeof(float) : 0;
    if (a.pattern_blocks + slices > 0) {
        cudaError_t err = allow_dynamic_smem((const void*)export_bsr_kernel, bytes);
        if (err != cudaSuccess) return err;
        export_bsr_kernel<<<a.pattern_blocks + slices, kExportThreads, bytes, s>>>(a);
    }
    if (values != nullptr && !narrow)
        export_columns_kernel<<<dim3(blocks_for(h.nslices, kExportWarps),
                                     std::min(65535, blocks_for(h.slice_width, kExportColumns))),
                                32 * kExportWarps, 0, s>>>(h.nslices, h.slice_ptr, h.slice_meta, h.row_info,
                                                           h.bsr_offsets, h.valA, h.valB, h.valC, values);
    return cudaGetLastError();
}

cudaError_t launch_export_triplets(Handle& h, float* values, cudaStream_t s) {
    if (h.ntrip == 0) return cudaSuccess;
    int threads = 256;
    int64_t blocks = (h.ntrip + threads - 1) / threads;
    export_triplets_kernel<<<(unsigned)blocks, threads, 0, s>>>(h.ntrip, h.trip_map, h.trip, values);
    return cudaGetLastError();
}

}  // namespace fem
