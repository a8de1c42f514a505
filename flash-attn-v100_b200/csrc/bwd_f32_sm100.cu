// Attention backward for fp32 inputs on the sm_100a tensor cores: every fp32 operand as three bf16 planes.
//
// The reference runs its backward's products of fp32 inputs through tl.dot with TF32 allowed
// (kernels/backward_kernel.py:118-176); one TF32 product misses this library's fp32 tolerance by more than an order
// of magnitude, so fp32 gradients were CUDA-core work: 1.27 ms of the 1.33 ms that forward + backward of B2 N1024
// H12 D64 causal took, at 9 TFLOP/s.  Here x = x1 + x2 + x3 with x1 = bf16(x), x2 = bf16(x - x1),
// x3 = bf16(x - x1 - x2): 24 significant bits, and bf16 has fp32's exponents, so no range is lost.  A product takes
// six of the nine partial products (those down to 2^-16 of the first); what is left out lies at 2^-25.  bf16 and not
// TF32 halves because six bf16 products cost what three TF32 ones do, a 16-bit tile serves as K-major and as MN-major
// operand alike (a 32-bit one would be needed twice), and three TF32 products stop at 2^-21.
//
// Accumulation.  The tensor core truncates when it adds to its fp32 accumulator, a bias that grows with every
// addition.  So the five small partial products of a contraction go first, while the accumulator is small, and no
// accumulator lives longer than one step: the step's dK, dV or dQ tile is added up in the threads' registers, where
// fp32 additions round to nearest.
//
// Three launches, all outputs owned by one CTA and summed in a fixed order:
//   1. split      Q, dO, K, V -> planes (p * B + b, N, H, 64); delta, lse padded
//   2. MODE 0     one CTA per 128-key tile, 64 queries a step:  S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
//   3. MODE 1     one CTA per 128-query tile, 64 keys a step:   S = Q K^T, dP = dO V^T, dQ += dS K
//
//   warps 0-15   a thread owns one TMEM lane (row of T1 / T2); warpgroup g owns the step's columns [16 g, 16 g + 16)
//   warp 16      MMA issuer      order  T1(0) T2(0) | T1(i+1) ACC2(i) T2(i+1) ACC1(i)
//   warp 17      TMA producer    (18, 19 idle)
// TMEM columns: T1 [0,64) and [448,512)  T2 [64,128)  P planes [128,224)  dS planes [224,320)  ACC1 [320,384)
// ACC2 [384,448).  T1 is two sums over half the head each: an error of a score is an error of P at full size.
// Shared memory: the stationary pair's planes 96 KB, two stages of the streamed pair's 96 KB, which is why head sizes
// above 64 stay on the CUDA cores.  Every mbarrier wait is bounded (sm100_ptx.cuh).
//
// What bounds it: the 96 (MODE 0) or 72 MMAs of 128 x 64 x 16 a step and the threads' splitting of P and dS (about 25
// instructions a score) are of the same length and overlap by one step.  B200, B2 N1024 H12 causal, CUDA cores -> here:
// delta / split 11 -> 17 us, dK and dV 749 -> 59 us, dQ 522 -> 48 us.
//
// Error against float64 (rel-L2 of dq, dk, dv, the largest of the three; forward and lse from the TF32 kernel), CUDA
// cores -> here: N2048 full 2.9e-6 -> 2.7e-6, N1024 causal 1.8e-6 -> 1.5e-6, with scores 16 times as large
// 6.1e-5 -> 5.8e-5.  From a forward without error it would be 1.0e-6 -> 5.2e-7, 8.0e-7 -> 3.8e-7 and 3.6e-6 -> 7.3e-6:
// inside one MMA the tensor core aligns sixteen products and drops what lies below, which shows when scores are large.
// So the rule takes the calls whose forward is the TF32 kernel (D = 64, aligned tensors, positive scale) and leaves the
// others, whose forward is as exact as the CUDA cores', where they were; a caller whose o and lse come from another
// forward offers no scratch.  An infinite operand (or one beyond bf16's largest value) gives NaN here where the
// CUDA-core kernels may give an infinity: its planes are inf, NaN, NaN.
#include "fa_common.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

namespace fa {
namespace {

using namespace ptx;

constexpr int kRows = 128;                    // stationary rows of a CTA
constexpr int kStep = 64;                     // streamed rows of a step
constexpr int kDim = 64;                      // columns of a plane
constexpr int kPlanes = 3;
constexpr int kStatPlane = kRows * 128, kStrmPlane = kStep * 128;        // bytes: rows of 64 bf16
constexpr int kStat = kPlanes * kStatPlane, kStrm = kPlanes * kStrmPlane;
constexpr int kWorkers = 16;                  // elementwise warps
constexpr int kThreads = 32 * (kWorkers + 4);
constexpr float kLog2e = 1.4426950408889634f;
// partial products, the small ones first: planes of the first and of the second operand
constexpr int kPairs = 6;
__device__ constexpr int kPairA[kPairs] = {0, 2, 1, 0, 1, 0};
__device__ constexpr int kPairB[kPairs] = {2, 0, 1, 1, 0, 0};

enum { kBarXY = 0, kBarU = 1 /*[2]*/, kBarW = 3 /*[2]*/, kBarUFree = 5 /*[2]*/, kBarWFree = 7 /*[2]*/, kBarT1 = 9, kBarT2 = 10,
       kBarAcc = 11, kBarT1Read = 12, kBarT2Read = 13, kBarP = 14, kBarDs = 15, kNumBars = 16 };
constexpr int kSmemBytes = 2 * kStat + 4 * kStrm + kNumBars * 8 + 64 + 1024;

struct F32Args {
    const float* lse;              // [B*H][nq_pad], +inf in the padding
    const float* delta;            // [B*H][nq_pad], 0 in the padding
    fa_b200_tensor out1, out2;     // MODE 0: dK, dV; MODE 1: dQ
    const int32_t* kv_len;
    int32_t* status;
    int B, Nq, Nk, H, Hkv, nq_pad;
    int causal, shift, vec, wait_limit_ms;
    float scale;
};

// x -> three bf16 planes, two values packed per word
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& a, uint32_t& b, uint32_t& c) {
    float h0, h1;
    auto less = [&] { f2_unpack(f2_fma(f2_pack(h0, h1), 0xBF800000BF800000ull, f2_pack(x0, x1)), x0, x1); };     // x -= h, both at once
    a = pack2<true>(x0, x1);
    unpack2<true>(a, h0, h1);
    less();
    b = pack2<true>(x0, x1);
    unpack2<true>(b, h0, h1);
    less();
    c = pack2<true>(x0, x1);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
bwd_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
               const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_w, const F32Args a) {
    constexpr bool KS = MODE == 0;             // key-stationary
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sX = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sY = sX + kStat;
    uint8_t* sU = sY + kStat;                  // two stages
    uint8_t* sW = sU + 2 * kStrm;              // two stages
    uint64_t* bars = (uint64_t*)(sW + 2 * kStrm);
    uint32_t* tmem_slot = (uint32_t*)(bars + kNumBars);
    volatile uint32_t* abort_flag = (volatile uint32_t*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // blocks start in linear order: columns fastest, the tiles with the most steps first
    const int cols = (int)(gridDim.y * gridDim.z);
    const int lin = (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
    const int rank = lin / cols, col = lin - rank * cols;
    const int tile = (!KS && a.causal) ? (int)gridDim.x - 1 - rank : rank;
    const int head_x = col % (int)gridDim.y, b = col / (int)gridDim.y;
    const int group = a.H / a.Hkv;
    const int nk = kv_len_of(a.kv_len, b, a.Nk);
    int it0 = 0, per_head, n_iter;
    if (KS) {
        if (a.causal && tile * kRows > a.shift) it0 = (tile * kRows - a.shift) / kStep;
        const int steps = (a.Nq + kStep - 1) / kStep;
        per_head = steps > it0 ? steps - it0 : 0;
        if (tile * kRows >= nk) per_head = 0;                    // padding keys: dK = dV = 0
        n_iter = per_head * group;
    } else {
        int kv_end = nk;
        if (a.causal && tile * kRows + kRows + a.shift < kv_end) kv_end = tile * kRows + kRows + a.shift;
        per_head = n_iter = (kv_end + kStep - 1) / kStep;
    }
    // streamed step `it`: its head and first row
    auto strm_head = [&](int it) { return KS ? head_x * group + it / per_head : head_x / group; };
    auto strm_row = [&](int it) { return (KS ? it0 + it % per_head : it) * kStep; };

    if (warp == 0) {
        if (lane < kNumBars) mbar_init(&bars[lane], lane >= kBarT1Read ? kWorkers : 1u);
        if (lane == 0) wait_control_init(abort_flag, a.wait_limit_ms);
        fence_mbar_init();
        __syncwarp();
    }
    if (warp == kWorkers) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == kWorkers + 1 && lane == 0) {
        prefetch_tensormap(&map_x); prefetch_tensormap(&map_y);
        prefetch_tensormap(&map_u); prefetch_tensormap(&map_w);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (KS) {
        grid_dependency_wait();                 // the planes: what stands above ran beside the end of the split kernel
        // The dQ kernel reads nothing the dK/dV kernel writes: it may take the SMs that this grid's last blocks leave idle
        // (launched serialized behind this grid, it waits for it only before it ends).  B2 N1024 H12 causal has 192 blocks
        // of 1 to 8 units in each.  The step at B4 N2048 H8 causal 538 -> 521 us, at B4 N1500 H8 without a mask 597 -> 587.
        grid_launch_dependents();
    }
    const uint32_t tmem = *tmem_slot;
    const uint32_t tT1 = tmem, tT2 = tmem + 64u, tP = tmem + 128u, tDs = tmem + 224u, tAcc1 = tmem + 320u, tAcc2 = tmem + 384u, tT1b = tmem + 448u;

    if (warp == kWorkers + 1) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one() && n_iter > 0) {
            mbar_expect_tx(&bars[kBarXY], 2 * kStat);
#pragma unroll
            for (int p = 0; p < kPlanes; ++p)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int at = p * kStatPlane + half * kStrmPlane, row = tile * kRows + half * kStep;
                    tma_load_4d(sX + at, &map_x, &bars[kBarXY], 0, head_x, row, p * a.B + b);
                    tma_load_4d(sY + at, &map_y, &bars[kBarXY], 0, head_x, row, p * a.B + b);
                }
            bool ok = true;
            int u_done = 0, w_done = 0;
            for (int it = 0; it < n_iter; ++it) {
                const int s = it & 1;
                const uint32_t ph = ((uint32_t)(it >> 1) & 1u) ^ 1u;
                const int head = strm_head(it), row = strm_row(it);
                ok = mbar_wait(&bars[kBarUFree + s], ph, abort_flag);
                if (!ok) break;
                mbar_expect_tx(&bars[kBarU + s], kStrm);
#pragma unroll
                for (int p = 0; p < kPlanes; ++p)
                    tma_load_4d(sU + s * kStrm + p * kStrmPlane, &map_u, &bars[kBarU + s], 0, head, row, p * a.B + b);
                ++u_done;
                ok = mbar_wait(&bars[kBarWFree + s], ph, abort_flag);
                if (!ok) break;
                mbar_expect_tx(&bars[kBarW + s], kStrm);
#pragma unroll
                for (int p = 0; p < kPlanes; ++p)
                    tma_load_4d(sW + s * kStrm + p * kStrmPlane, &map_w, &bars[kBarW + s], 0, head, row, p * a.B + b);
                ++w_done;
            }
            if (!ok) {
                // unwinding: let the copies in flight land before shared memory is given up
                for (int s = 0; s < 2; ++s) {
                    const int nu = (u_done + 1 - s) / 2, nw = (w_done + 1 - s) / 2;
                    for (int spin = 0; spin < 4096 && nu > 0 && !mbar_try_wait(&bars[kBarU + s], (uint32_t)(nu - 1) & 1u); ++spin) {}
                    for (int spin = 0; spin < 4096 && nw > 0 && !mbar_try_wait(&bars[kBarW + s], (uint32_t)(nw - 1) & 1u); ++spin) {}
                }
                for (int spin = 0; spin < 4096 && !mbar_try_wait(&bars[kBarXY], 0u); ++spin) {}
            }
        }
        __syncwarp();
    } else if (warp == kWorkers) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one() && n_iter > 0) {
            constexpr uint32_t idesc_t = make_idesc_f16(true, true, kRows, kStep, false, false);
            constexpr uint32_t idesc_acc = make_idesc_f16(true, true, kRows, kDim, false, true);
            const uint64_t dk_major = make_smem_desc_sw128(0, 0, 1024), dmn_major = make_smem_desc_sw128(0, 8192, 1024);
            const uint32_t sX_u = smem_u32(sX), sY_u = smem_u32(sY), sU_u = smem_u32(sU), sW_u = smem_u32(sW);
            // T = stationary x streamed^T over the 64 columns of the head
            auto issue_t = [&](uint32_t d_tmem, uint32_t stat_u, uint32_t strm_u, int k0, int k1) {
                const uint64_t a0 = dk_major + (uint64_t)(stat_u >> 4), b0 = dk_major + (uint64_t)(strm_u >> 4);
#pragma unroll
                for (int pr = 0; pr < kPairs; ++pr)
#pragma unroll
                    for (int kk = k0; kk < k1; ++kk)
                        mma_ss_f16(d_tmem, a0 + (uint64_t)((kPairA[pr] * kStatPlane + kk * 32) >> 4),
                                   b0 + (uint64_t)((kPairB[pr] * kStrmPlane + kk * 32) >> 4), idesc_t, (pr > 0 || kk > k0) ? 1u : 0u);
            };
            // ACC = A[TMEM planes] x streamed tile read MN-major, over the step's 64 streamed rows
            auto issue_acc = [&](uint32_t d_tmem, uint32_t a_tmem, uint32_t strm_u) {
                const uint64_t b0 = dmn_major + (uint64_t)(strm_u >> 4);
#pragma unroll
                for (int pr = 0; pr < kPairs; ++pr)
#pragma unroll
                    for (int kk = 0; kk < kStep / 16; ++kk)
                        mma_ts_f16(d_tmem, a_tmem + (uint32_t)(kPairA[pr] * 32 + kk * 8),
                                   b0 + (uint64_t)((kPairB[pr] * kStrmPlane + kk * 2048) >> 4), idesc_acc, (pr > 0 || kk > 0) ? 1u : 0u);
            };
            bool ok = mbar_wait(&bars[kBarXY], 0u, abort_flag);
            if (ok) ok = mbar_wait(&bars[kBarU], 0u, abort_flag);
            if (ok) ok = mbar_wait(&bars[kBarW], 0u, abort_flag);
            if (ok) {
                tc_fence_after_sync();
                issue_t(tT1, sX_u, sU_u, 0, 2);
                issue_t(tT1b, sX_u, sU_u, 2, 4);
                mma_commit(&bars[kBarT1]);
                issue_t(tT2, sY_u, sW_u, 0, 4);
                mma_commit(&bars[kBarT2]);
            }
            for (int it = 0; it < n_iter && ok; ++it) {
                const int s = it & 1, ns = s ^ 1;
                const uint32_t ph = (uint32_t)it & 1u, nph = (uint32_t)((it + 1) >> 1) & 1u;
                const bool more = it + 1 < n_iter;
                if (more) {
                    ok = mbar_wait(&bars[kBarT1Read], ph, abort_flag);
                    if (ok) ok = mbar_wait(&bars[kBarU + ns], nph, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    issue_t(tT1, sX_u, sU_u + ns * kStrm, 0, 2);
                    issue_t(tT1b, sX_u, sU_u + ns * kStrm, 2, 4);
                    mma_commit(&bars[kBarT1]);
                }
                // P(it) is in its planes, and the sums of step it - 1 have been read
                ok = mbar_wait(&bars[kBarP], ph, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                if (KS) issue_acc(tAcc2, tP, sW_u + s * kStrm);
                if (more) {
                    ok = mbar_wait(&bars[kBarT2Read], ph, abort_flag);
                    if (ok) ok = mbar_wait(&bars[kBarW + ns], nph, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    issue_t(tT2, sY_u, sW_u + ns * kStrm, 0, 4);
                    mma_commit(&bars[kBarT2]);
                }
                ok = mbar_wait(&bars[kBarDs], ph, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                issue_acc(tAcc1, tDs, sU_u + s * kStrm);
                mma_commit(&bars[kBarAcc]);
                mma_commit(&bars[kBarUFree + s]);
                mma_commit(&bars[kBarWFree + s]);
            }
        }
        __syncwarp();
    } else if (warp < kWorkers) {
        // ------------------------------------------------------------ P, dS, sums, epilogue
        const int g = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const int row = tile * kRows + r;              // key (MODE 0) or query (MODE 1)
        float my_lse = 0.f, my_delta = 0.f;
        if (!KS) {
            const int64_t at = ((int64_t)b * a.H + head_x) * a.nq_pad + row;
            my_lse = a.lse[at];
            my_delta = a.delta[at];
        }
        float acc1[16], acc2[KS ? 16 : 1];
#pragma unroll
        for (int c = 0; c < 16; ++c) { acc1[c] = 0.f; if (KS) acc2[c] = 0.f; }
        // the sums of a finished step, from tensor memory into the registers
        auto fold = [&] {
            uint32_t x[16];
            tmem_ld_32x16(tAcc1 + lane_off + (uint32_t)(16 * g), x);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c) acc1[c] += __uint_as_float(x[c]);
            if constexpr (KS) {
                tmem_ld_32x16(tAcc2 + lane_off + (uint32_t)(16 * g), x);
                tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 16; ++c) acc2[c] += __uint_as_float(x[c]);
            }
        };
        // 16 values -> the three planes of my row and columns
        auto store_planes = [&](uint32_t t, const float (&x)[16]) {
            uint32_t pa[8], pb[8], pc[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) split3(x[2 * c], x[2 * c + 1], pa[c], pb[c], pc[c]);
            const uint32_t at = t + lane_off + (uint32_t)(8 * g);
            tmem_st_32x8(at, pa);
            tmem_st_32x8(at + 32u, pb);
            tmem_st_32x8(at + 64u, pc);
            tmem_wait_st();
            tc_fence_before_sync();
        };
        bool ok = true;
        for (int it = 0; it < n_iter; ++it) {
            const uint32_t ph = (uint32_t)it & 1u;
            const int col0 = strm_row(it) + 16 * g;    // my first streamed row: query (MODE 0) or key (MODE 1)
            const int64_t at = KS ? ((int64_t)b * a.H + strm_head(it)) * a.nq_pad + col0 : 0;
            float v[16];                               // lse, then delta of my columns' queries, asked for ahead of the waits
            auto load_v = [&](const float* src) {
#pragma unroll
                for (int c = 0; c < 16; c += 4) {
                    const float4 f = *reinterpret_cast<const float4*>(src + at + c);
                    v[c] = f.x; v[c + 1] = f.y; v[c + 2] = f.z; v[c + 3] = f.w;
                }
            };
            if (KS) load_v(a.lse);
            ok = mbar_wait(&bars[kBarT1], ph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            uint32_t t1[16], t1b[16];
            tmem_ld_32x16(tT1 + lane_off + (uint32_t)(16 * g), t1);
            tmem_ld_32x16(tT1b + lane_off + (uint32_t)(16 * g), t1b);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[kBarT1Read]);
            float p[16];
            // the difference is rounded once and small wherever P is not: base 2 comes after it
#pragma unroll
            for (int c = 0; c < 16; ++c) p[c] = ex2(fmaf(__uint_as_float(t1[c]) + __uint_as_float(t1b[c]), a.scale, -(KS ? v[c] : my_lse)) * kLog2e);
            if (KS) {
                const int hidden = a.causal ? row - a.shift - col0 : 0;       // my first columns do not see the key
#pragma unroll
                for (int c = 0; c < 16; ++c) if (c < hidden || row >= nk) p[c] = 0.f;
                load_v(a.delta);
            } else {
                int seen = nk - col0;
                if (a.causal && row + a.shift + 1 - col0 < seen) seen = row + a.shift + 1 - col0;
#pragma unroll
                for (int c = 0; c < 16; ++c) if (c >= seen) p[c] = 0.f;
            }
            if (it > 0) {
                ok = mbar_wait(&bars[kBarAcc], ph ^ 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after_sync();
                fold();
                tc_fence_before_sync();
            }
            if (KS) store_planes(tP, p);
            mbar_arrive_warp(&bars[kBarP]);
            ok = mbar_wait(&bars[kBarT2], ph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            uint32_t t2[16];
            tmem_ld_32x16(tT2 + lane_off + (uint32_t)(16 * g), t2);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[kBarT2Read]);
#pragma unroll
            for (int c = 0; c < 16; ++c) p[c] *= __uint_as_float(t2[c]) - (KS ? v[c] : my_delta);
            store_planes(tDs, p);
            mbar_arrive_warp(&bars[kBarDs]);
        }
        if (n_iter > 0 && ok) {
            ok = mbar_wait(&bars[kBarAcc], (uint32_t)(n_iter - 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                tc_fence_after_sync();
                fold();
            }
        }
        if (ok && row < (KS ? a.Nk : a.Nq)) {
            auto put = [&](const fa_b200_tensor& t, const float (&x)[16], float mul) {
                float* dst = (float*)t.ptr + (int64_t)b * t.stride_b + (int64_t)row * t.stride_n + (int64_t)head_x * t.stride_h + 16 * g;
                if (a.vec) {
#pragma unroll
                    for (int c = 0; c < 16; c += 4)
                        *reinterpret_cast<float4*>(dst + c) = make_float4(x[c] * mul, x[c + 1] * mul, x[c + 2] * mul, x[c + 3] * mul);
                } else {
#pragma unroll
                    for (int c = 0; c < 16; ++c) dst[c] = x[c] * mul;
                }
            };
            put(a.out1, acc1, a.scale);
            if constexpr (KS) put(a.out2, acc2, 1.f);
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWorkers) tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0 && *abort_flag) report_status(a.status, 6 + MODE);
    if (!KS) grid_dependency_wait();            // the end of this grid must still mean the end of the dK/dV grid
}

// Planes of the four operands, delta and the padded lse.  Eight lanes share a row, eight columns each: 32 bytes of an fp32
// operand come in two loads, 16 bytes go to each plane.  Rows [0, q_rows) are (batch, padded query, head), the rest (batch,
// key, K/V head), heads fastest as in memory.  Bound by the stores: B2 N1024 H12 is 25 MB in (31 with o) and 38 MB out.  One
// warp a row with 4-byte accesses and 64-bit divisions took 17.2 us there, this 9.3.
struct SplitArgs {
    fa_b200_tensor q, k, v, o, d_o;
    const float* lse_in;
    uint32_t *q16, *g16, *k16, *v16;      // planes, two columns per word
    float *lse, *delta;
    int B, Nq, Nk, H, Hkv, nq_pad;
    uint32_t q_rows, rows;
    int vec_q, vec_kv;                    // their rows can be read as float4
};
__global__ void __launch_bounds__(256) bwd_f32_split_kernel(const SplitArgs a) {
    grid_launch_dependents();
    const uint32_t sub = threadIdx.x & 7u, row = blockIdx.x * 32u + (threadIdx.x >> 3);
    const bool in = row < a.rows;
    auto load = [&](const fa_b200_tensor& t, bool vec, uint32_t b, uint32_t n, uint32_t h, float (&x)[8]) {
        const float* src = (const float*)t.ptr + b * t.stride_b + n * t.stride_n + h * t.stride_h + sub * 8;
        if (vec) {
            const float4 lo = reinterpret_cast<const float4*>(src)[0], hi = reinterpret_cast<const float4*>(src)[1];
            x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w; x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = src[e];
        }
    };
    auto store = [&](uint32_t* dst, uint32_t N, uint32_t H, uint32_t b, uint32_t n, uint32_t h, const float (&x)[8]) {
        uint32_t p[kPlanes][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3(x[2 * e], x[2 * e + 1], p[0][e], p[1][e], p[2][e]);
#pragma unroll
        for (int i = 0; i < kPlanes; ++i)
            *reinterpret_cast<uint4*>(dst + ((((int64_t)i * a.B + b) * N + n) * H + h) * (kDim / 2) + sub * 4) =
                make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
    };
    float x[8], y[8];
    float s = 0.f;                         // (every lane takes part in the sum below)
    int64_t at = -1;
    if (in && row < a.q_rows) {
        const uint32_t rest = row / (uint32_t)a.H, h = row - rest * (uint32_t)a.H, b = rest / (uint32_t)a.nq_pad, i = rest - b * (uint32_t)a.nq_pad;
        const int64_t out = ((int64_t)b * a.H + h) * a.nq_pad + i;
        if (i >= (uint32_t)a.Nq) {
            if (sub == 0) { a.lse[out] = INFINITY; a.delta[out] = 0.f; }
        } else {
            at = out;
            load(a.q, a.vec_q, b, i, h, x);
            store(a.q16, a.Nq, a.H, b, i, h, x);
            load(a.d_o, a.vec_q, b, i, h, x);
            load(a.o, a.vec_q, b, i, h, y);
            store(a.g16, a.Nq, a.H, b, i, h, x);
            s = (fmaf(x[0], y[0], x[1] * y[1]) + fmaf(x[2], y[2], x[3] * y[3])) + (fmaf(x[4], y[4], x[5] * y[5]) + fmaf(x[6], y[6], x[7] * y[7]));
            if (sub == 0) a.lse[out] = a.lse_in[((int64_t)b * a.H + h) * a.Nq + i];
        }
    } else if (in) {
        const uint32_t kr = row - a.q_rows, rest = kr / (uint32_t)a.Hkv, h = kr - rest * (uint32_t)a.Hkv, b = rest / (uint32_t)a.Nk,
                       j = rest - b * (uint32_t)a.Nk;
        load(a.k, a.vec_kv, b, j, h, x);
        load(a.v, a.vec_kv, b, j, h, y);
        store(a.k16, a.Nk, a.Hkv, b, j, h, x);
        store(a.v16, a.Nk, a.Hkv, b, j, h, y);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (at >= 0 && sub == 0) a.delta[at] = s;
}

struct F32Layout { size_t q, g, k, v, lse, delta, bytes; };
F32Layout f32_layout(const fa_b200_params& p) {
    F32Layout l;
    size_t at = 0;
    auto region = [&](size_t n) { const size_t r = at; at = align_up(at + n, 256); return r; };
    const size_t q = (size_t)kPlanes * p.B * p.Nq * p.H * kDim * 2, k = (size_t)kPlanes * p.B * p.Nk * p.Hkv * kDim * 2;
    const size_t rows = (size_t)p.B * p.H * align_up((size_t)p.Nq, 128) * sizeof(float);
    l.q = region(q); l.g = region(q); l.k = region(k); l.v = region(k); l.lse = region(rows); l.delta = region(rows);
    l.bytes = at;
    return l;
}

}  // namespace

// Which backward calls the planes serve, and the scratch they take (0: not served): those whose forward the TF32 kernel
// serves (kernel comment).  Other head sizes, a bias, dropout and tensors that kernel refuses stay on the CUDA cores.
size_t sm100_f32_bwd_scratch_bytes(const fa_b200_params& p) {
    if (p.dtype != FA_B200_F32 || p.variant != FA_B200_VARIANT_AUTO || p.D != kDim) return 0;
    const char* why = "";
    if (p.d_scores || !sm100_tf32_fwd_supports(p, &why)) return 0;
    if (p.B > 65535 / kPlanes || p.H > 65535 || p.B < 1 || p.Nq < 1 || p.Nk < 1) return 0;
    return f32_layout(p).bytes;
}

int sm100_f32_bwd(const fa_b200_params& p, void* scratch) {
    const F32Layout l = f32_layout(p);
    char* ws = (char*)scratch;
    cudaStream_t st = (cudaStream_t)p.stream;
    const int nq_pad = (int)align_up((size_t)p.Nq, 128);
    const int phases = p.bwd_phases ? p.bwd_phases : 7;
    auto aligned = [&](const fa_b200_tensor& t) {
        return ((uintptr_t)t.ptr & 15u) == 0 && t.stride_b % 4 == 0 && t.stride_n % 4 == 0 && t.stride_h % 4 == 0;
    };
    if (phases & 1) {
        SplitArgs s;
        s.q = p.q; s.k = p.k; s.v = p.v; s.o = p.o; s.d_o = p.d_o; s.lse_in = p.lse;
        s.q16 = (uint32_t*)(ws + l.q); s.g16 = (uint32_t*)(ws + l.g); s.k16 = (uint32_t*)(ws + l.k); s.v16 = (uint32_t*)(ws + l.v);
        s.lse = (float*)(ws + l.lse); s.delta = (float*)(ws + l.delta);
        s.B = p.B; s.Nq = p.Nq; s.Nk = p.Nk; s.H = p.H; s.Hkv = p.Hkv; s.nq_pad = nq_pad;
        const int64_t q_rows = (int64_t)p.B * nq_pad * p.H, rows = q_rows + (int64_t)p.B * p.Nk * p.Hkv;
        if (rows > 0x7fffffff) { set_error("problem too large for the split grid"); return FA_EUNSUPPORTED; }
        s.q_rows = (uint32_t)q_rows; s.rows = (uint32_t)rows;
        s.vec_q = aligned(p.q) && aligned(p.o) && aligned(p.d_o); s.vec_kv = aligned(p.k) && aligned(p.v);
        bwd_f32_split_kernel<<<(unsigned)((rows + 31) / 32), 256, 0, st>>>(s);
        FA_CUDA_CHECK(cudaGetLastError());
    }
    CUtensorMap mq, mg, mk, mv;
    int r;
    auto planes = [&](CUtensorMap* m, size_t off, int N, int H) {
        return cached_tmap_bnhd(m, ws + off, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (int64_t)kPlanes * p.B, N, H, kDim, (int64_t)N * H * kDim,
                                (int64_t)H * kDim, (int64_t)kDim, kStep, 64, 1);
    };
    if ((r = planes(&mq, l.q, p.Nq, p.H)) || (r = planes(&mg, l.g, p.Nq, p.H)) ||
        (r = planes(&mk, l.k, p.Nk, p.Hkv)) || (r = planes(&mv, l.v, p.Nk, p.Hkv))) {
        set_error("cuTensorMapEncodeTiled failed (%d)", r);
        return FA_ECUDA;
    }
    F32Args a;
    a.lse = (const float*)(ws + l.lse); a.delta = (const float*)(ws + l.delta);
    a.kv_len = p.kv_lengths; a.status = p.status_word;
    a.B = p.B; a.Nq = p.Nq; a.Nk = p.Nk; a.H = p.H; a.Hkv = p.Hkv; a.nq_pad = nq_pad;
    a.causal = p.causal; a.shift = p.causal ? p.causal_shift : 0;
    a.wait_limit_ms = p.wait_limit_ms;
    a.scale = p.scale;
    {
        static std::mutex mu;
        static uint64_t done[2] = {0, 0};
        FA_CUDA_CHECK(set_smem_limit_once(bwd_f32_kernel<0>, kSmemBytes, p.device, &done[0], &mu));
        FA_CUDA_CHECK(set_smem_limit_once(bwd_f32_kernel<1>, kSmemBytes, p.device, &done[1], &mu));
    }
    if (phases & 2) {
        a.out1 = p.dk; a.out2 = p.dv;
        a.vec = aligned(p.dk) && aligned(p.dv);
        const dim3 grid((p.Nk + kRows - 1) / kRows, p.Hkv, p.B);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid; cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmemBytes; cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = (phases & 1) ? 1 : 0;        // only behind the split kernel of this call
        FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, bwd_f32_kernel<0>, mk, mv, mq, mg, a));
    }
    if (phases & 4) {
        a.out1 = p.dq; a.out2 = p.dq;
        a.vec = aligned(p.dq);
        const dim3 grid((p.Nq + kRows - 1) / kRows, p.H, p.B);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid; cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmemBytes; cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = (phases & 2) ? 1 : 0;        // only behind the dK/dV kernel of this call
        FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, bwd_f32_kernel<1>, mq, mg, mk, mv, a));
    }
    return FA_OK;
}

}  // namespace fa
