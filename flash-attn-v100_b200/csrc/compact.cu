// Kept keys first: the order of a boolean key-padding mask, and rows moved by it.
//
// The attention layer turns a padding mask into per-batch key counts by moving every entry's kept keys to the front
// (the reference expands the mask to a dense (B, H, Nq, Nk) bias instead, examples/basic_usage.py:228-250).  As torch
// operations that is a sort, a handful of element-wise launches, two gathers that read an index per element, and two
// zero-fills and scatters in the backward: 0.29 ms of the 1.29 ms of a layer's step at B16 N1000 H16 D64 bf16.
// Here: one scan per batch entry and one launch that moves whole rows of K and V, 16 bytes a thread, each way.
// Bound by memory: K and V read and written once, 131 MB at that size, 20 us at the copy rate.
#include "fa_common.cuh"

namespace fa {
namespace {

constexpr int kScanThreads = 1024;

// order[b][p] = key that comes p-th: the keys with mask 0 in their order, then the others in theirs (a stable sort).
// One block per batch entry, two passes over its mask (their number, then their places).
__global__ void __launch_bounds__(kScanThreads) key_order_kernel(const uint8_t* __restrict__ mask, int64_t mask_stride_b, int N,
                                                                 int* __restrict__ order, int* __restrict__ counts) {
    __shared__ int warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint8_t* m = mask + (int64_t)blockIdx.x * mask_stride_b;
    int* dst = order + (int64_t)blockIdx.x * N;
    // sum over the block of the warps' numbers; `before`: those of the warps in front of mine
    auto block_sum = [&](int v, int& before) {
        __syncthreads();                               // the previous round's values have been read
        if (lane == 0) warp_sum[warp] = v;
        __syncthreads();
        int x = warp_sum[lane];
        before = __reduce_add_sync(0xffffffffu, lane < warp ? x : 0);
        return __reduce_add_sync(0xffffffffu, x);
    };
    int mine = 0, unused;
    for (int j = threadIdx.x; j < N; j += kScanThreads) mine += m[j] == 0;
    const int kept = block_sum(__reduce_add_sync(0xffffffffu, mine), unused);
    int done = 0;                                      // kept keys of the rounds before
    for (int j0 = 0; j0 < N; j0 += kScanThreads) {
        const int j = j0 + (int)threadIdx.x;
        const bool keep = j < N && m[j] == 0;
        const uint32_t bits = __ballot_sync(0xffffffffu, keep);
        int before;
        const int total = block_sum(__popc(bits), before);
        const int rank = done + before + __popc(bits & ((1u << lane) - 1u));        // kept keys in front of j
        if (j < N) dst[keep ? rank : kept + (j - rank)] = j;
        done += total;
    }
    if (threadIdx.x == 0) counts[blockIdx.x] = kept > 0 ? kept : 1;
}

// gather: dst[b][p] = src[b][order[b][p]];  scatter: dst[b][order[b][p]] = src[b][p].  Dense rows of `pieces` 16-byte
// pieces; two tensors of one shape (blockIdx.y).
template <bool SCATTER>
__global__ void __launch_bounds__(256) permute_rows_kernel(const uint4* s0, const uint4* s1, uint4* d0, uint4* d1,
                                                           const int* __restrict__ order, uint32_t N, uint32_t pieces, uint32_t total) {
    const uint4* src = blockIdx.y ? s1 : s0;
    uint4* dst = blockIdx.y ? d1 : d0;
    // four pieces a thread, a block's width apart, all loads ahead of the stores
    const uint32_t first = blockIdx.x * 1024u + threadIdx.x;
    uint4 x[4];
    uint32_t to[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const uint32_t at = first + e * 256u;
        to[e] = 0xFFFFFFFFu;
        if (at >= total) continue;
        const uint32_t row = at / pieces;              // b * N + p
        const uint32_t other = (row / N * N + (uint32_t)order[row]) * pieces + (at - row * pieces);
        to[e] = SCATTER ? other : at;
        x[e] = src[SCATTER ? at : other];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) if (to[e] != 0xFFFFFFFFu) dst[to[e]] = x[e];
}

}  // namespace
}  // namespace fa

using namespace fa;

extern "C" {

int fa_b200_key_order(const uint8_t* mask, int64_t mask_stride_b, int B, int N, int32_t* order, int32_t* counts, int device, void* stream) {
    if (B < 0 || N < 0) { set_error("key_order: negative size"); return FA_EINVAL; }
    if (B == 0) return FA_OK;
    if (!counts || (N > 0 && (!mask || !order))) { set_error("key_order: null pointer"); return FA_EINVAL; }
    GuardDevice g(device);
    if (!g.ok) { set_error("cudaSetDevice(%d) failed", device); return FA_ECUDA; }
    key_order_kernel<<<(unsigned)B, kScanThreads, 0, (cudaStream_t)stream>>>(mask, mask_stride_b, N, order, counts);
    FA_CUDA_CHECK(cudaGetLastError());
    return FA_OK;
}

int fa_b200_permute_rows(const void* src0, const void* src1, void* dst0, void* dst1, const int32_t* order, int B, int N,
                         size_t row_bytes, int scatter, int device, void* stream) {
    if (B < 0 || N < 0) { set_error("permute_rows: negative size"); return FA_EINVAL; }
    if (B == 0 || N == 0 || row_bytes == 0) return FA_OK;
    if (!src0 || !src1 || !dst0 || !dst1 || !order) { set_error("permute_rows: null pointer"); return FA_EINVAL; }
    if (row_bytes % 16 != 0 || row_bytes / 16 > 0x7fffffff ||
        (((uintptr_t)src0 | (uintptr_t)src1 | (uintptr_t)dst0 | (uintptr_t)dst1) & 15u) != 0) {
        set_error("permute_rows: rows must be 16-byte aligned and a multiple of 16 bytes");
        return FA_EALIGN;
    }
    const uint32_t pieces = (uint32_t)(row_bytes / 16);
    const double all = (double)B * (double)N * (double)pieces;
    if (all > 4294960000.0) { set_error("permute_rows: more than 2^32 pieces of 16 bytes"); return FA_EUNSUPPORTED; }
    const uint32_t total = (uint32_t)B * (uint32_t)N * pieces, blocks = (uint32_t)(((uint64_t)total + 1023) / 1024);
    GuardDevice g(device);
    if (!g.ok) { set_error("cudaSetDevice(%d) failed", device); return FA_ECUDA; }
    const dim3 grid(blocks, 2);
    auto kernel = scatter ? permute_rows_kernel<true> : permute_rows_kernel<false>;
    kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint4*)src0, (const uint4*)src1, (uint4*)dst0, (uint4*)dst1, order, (uint32_t)N, pieces, total);
    FA_CUDA_CHECK(cudaGetLastError());
    return FA_OK;
}

}  // extern "C"
