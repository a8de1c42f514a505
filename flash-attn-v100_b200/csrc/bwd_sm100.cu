// Attention backward for sm_100a: TMA -> shared memory -> tcgen05.mma with
// accumulators in tensor memory, warp-specialised.
//
// Replaces the reference's Triton backward kernel
// (kernels/backward_kernel.py:17-205) and its launcher (:208-318).
//
// Three launches:
//   1. preprocess  -delta = -rowsum(dO o O) and -lse*log2(e), both fp32, written
//                  to the workspace in rows padded to whole 128-row tiles
//                  (padding: delta = 0, -lse = -inf, so padded queries get P = 0)
//   2. MODE 0      a block is a 128-row key tile (stationary K, V), streams the
//                  query tiles: writes dK and dV
//   3. MODE 1      a block is a 128-row query tile (stationary Q, dO), streams
//                  the key tiles: writes dQ
// 2 starts beside the end of 1 and waits for it before it reads; 3 may run beside the end of 2 (griddepcontrol).
// Every output element is owned by one block and accumulated in a fixed order, so
// results are bit-reproducible (the reference accumulates dQ across CTAs with
// an unordered read-modify-write, kernels/backward_kernel.py:179-194).
//
// D = 64 has a faster route (MODE 2) unless the two-pass variant is asked for:
// the key-stationary kernel also forms the step's dQ tile, dS K_j, from the
// dS^T tile its threads leave in shared memory, and adds it to an fp32 buffer in
// global memory (red.global.add.v4.f32, order across CTAs not fixed); S and dP
// are then computed once instead of twice.  Launches: memset of the buffer +
// preprocess, MODE 2, and a conversion of the sums to dQ.  At D = 128 tensor
// memory has no columns left for the dQ tile and the additions cost more than
// the second kernel's recomputation, so that size keeps the two passes.
//
// Both modes run the same pipeline on a stationary pair (X, Y) and a streamed
// pair (U, W):
//                         MODE 0 (dK, dV)          MODE 1 (dQ)
//   X, Y                  K_j, V_j                 Q_i, dO_i
//   U, W                  Q_i, dO_i                K_j, V_j
//   T1 = X U^T            S^T                      S
//   T2 = Y W^T            dP^T                     dP
//   phase A (T1 -> P)     P^T = exp2(S^T c - lse)  P = exp2(S c - lse)
//   phase B (T2 -> dS)    dS^T = P^T o (dP^T o Z - delta)
//   ACC2 += P  W          dV += (P o Z)^T dO       (not computed)
//   ACC1 += dS U          dK += dS^T Q             dQ += dS K
// T1/T2 are SS MMAs (both operands K-major in shared memory); the accumulating
// MMAs take P / dS from TMEM (written over T1 / T2 by the threads that read
// them) and U / W from the same shared-memory tiles read MN-major.
//
//   warps 0-15       four elementwise warpgroups; a thread owns one TMEM lane (row)
//                    and warpgroup g owns columns [32g, 32g+32) of T1/T2
//   warp 16          MMA issuer; order  T1(0) T2(0) | ACC2(i) T1(i+1) ACC1(i) T2(i+1) ...  (MODE 0, 2)
//                                       T1(0) T2(0) | T1(i+1) T2(i+1) ACC1(i) ...          (MODE 1)
//   warp 17          TMA producer: U and W tiles into rings of their own (U is read again by the
//                    step's last MMA, so it gets three stages where shared memory allows and its
//                    next load overlaps a whole step; W gets two), and in the key-stationary
//                    kernels the step's -lse / -delta rows into a two-slot ring
//   warp 18          calls with a bias: brings the steps' bias tiles (TMA)
//   warp 19          stores by TMA: the fp16 copy of K, and each block's results once they are staged
//   warps 18-19      INLINE: convert the streamed tiles to fp16 in place as they land (all MMAs run f16 x f16, with P
//                    and dS rounded to fp16; see "number formats" below); stationary tiles: the elementwise warps do
//
// A CTA goes on from one block of the grid to the next: the producer asks for another block (clusterlaunchcontrol: the
// answer is a block that has not been started, so the order of the grid and its balance stay what they are) when it
// begins one, and leaves its place for the other warps in one of two slots.  Nothing is set up again; the rings, their
// phases and tensor memory carry on.  The next block's X, U, W and its first products come while the last one's results
// are still read out: those go to shared memory (dK or dQ over the block's last U tile, dV over its last W tile, by then
// read by every MMA) and leave by TMA.  B32 N197 H12 D64 fp16: dK/dV and dQ 46 and 40 -> 30 and 24
// us; backward alone under a sustained load, B8 N2048 H16 D64 fp16 688 -> 620, B4 N4096 H32 D128 bf16 causal 2011 -> 1871,
// B1 N16384 H32 D128 6244 -> 6197 (there the board's power limit sets the pace).
// Stored straight from registers, the results took 2200-6000 cycles a block.
//
// TMEM columns: T1 [0,128)  T2 [128,256)  ACC1 [256,256+D)  ACC2 [384,384+D).
// MODE 1 has no ACC2 and never writes P back (only dS is an MMA operand there): S has the one buffer
// T1, free again once the threads hold S(i) in registers, and dP / dS alternate between T2 and
// [384,512), so that S(i+1) and dP(i+1) are both computed while the threads work on step i.
// MODE 2 (D = 64) puts the dQ tile at [448,512).
// Every mbarrier wait is bounded; see sm100_ptx.cuh.
#include "fa_common.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"
#include "tile_config.cuh"
#include <type_traits>

namespace fa {
namespace {

using namespace ptx;

constexpr int kTile = 128;
constexpr int kBoxBytes = 128 * 128;
constexpr int kNWG = tile::kBwdWarpgroups;   // elementwise warpgroups per CTA (each owns 128 / kNWG columns)
constexpr int kExtraThreads = 128;       // MMA warp, TMA warp, warps 18 and 19: registers are granted per four warps
constexpr float kLog2e = 1.4426950408889634f;

// Shared-memory plan of one kernel instance.  The streamed tiles U and W have rings of their own:
// U (Q_i in the key-stationary kernels, K_j in MODE 1) is read by the first MMA of its step and again
// by the last one, a step and a half later, so two stages leave the TMA load of the next tile no
// time at all (it can only start when the last reader has finished and is needed at once); W is
// done within one step.  D = 128 has room for three U stages and two W stages, except that the
// key-stationary dropout instance needs 4 KB for its masks and stays at two and two.
// DROP: 0 no dropout; 1 keep bits drawn by the kernel's own threads; 2 loaded from the call's bit buffer.
// PREC: 0 for calls with D = 64 or 128; 1 ("pair") for 16-bit calls with an additive bias or another head size (any
// multiple of 8 up to 128, the tiles padded by TMA's zero fill): P and dS go back to tensor memory as hi + lo in the
// inputs' own format and every accumulating MMA is issued for both, so they keep 17 (bf16) or 22 (fp16) significant
// bits and no operand is converted.  2: the same with the step's 128 x 128 bias tile brought to shared memory by TMA
// (see the forward; here the key-stationary kernel would read a value, the other one 16 bytes of 32 lines, per load).
template <int D, int MODE, int DROP, int PREC>
struct BwdCfg {
    static constexpr int kNBox = D / 64;
    static constexpr int kTileBytes = kNBox * kBoxBytes;
    static constexpr bool kFused = (MODE == 2);
    static constexpr bool kMasks = DROP == 1 && MODE != 1;       // masks are built in shared memory when keys are rows
    static constexpr int kUStages = PREC == 2 ? tile::bwd_bias_u_stages(D) : tile::bwd_u_stages(D, kMasks);
    static constexpr int kWStages = PREC == 2 ? tile::bwd_bias_w_stages(D) : tile::bwd_w_stages(D);
    static constexpr int kBiasBytes = PREC == 2 ? 4 * kBoxBytes : 0;    // four boxes of 128 queries x 32 keys
    static constexpr int kMaskBytes = 2 * 128 * 8 * 2;          // two buffers of 128 x 8 uint16 keep masks
    static constexpr int kXFull = 0;
    static constexpr int kYFull = 1;
    static constexpr int kXEmpty = 2;                            // the item's last reader of X (the MMAs; with a copy of K its store, too)
    static constexpr int kYEmpty = 3;
    static constexpr int kSchedFull = 4;                         // [2] the next item's place is in its slot
    static constexpr int kSchedEmpty = 6;                        // [2] ... and has been read (one arrival per reading warp)
    static constexpr int kClc = 8;                               // the answer to the request for another item has landed
    static constexpr int kUFull = 9;                             // [kUStages]
    static constexpr int kUEmpty = kUFull + kUStages;            // [kUStages]
    static constexpr int kWFull = kUEmpty + kUStages;            // [kWStages]
    static constexpr int kWEmpty = kWFull + kWStages;            // [kWStages]
    static constexpr int kT1Full = kWEmpty + kWStages;           // [2]: one per S buffer (MODE 0 uses the first)
    static constexpr int kT2Full = kT1Full + 2;
    static constexpr int kPReady = kT2Full + 1;                  // one arrival per elementwise warp
    static constexpr int kDsReady = kPReady + 1;                 // one arrival per elementwise warp
    static constexpr int kAccDone = kDsReady + 1;
    static constexpr int kMask = kAccDone + 1;                   // one arrival per elementwise warp
    static constexpr int kEpi = kMask + 1;                       // one arrival per elementwise warp: results are staged
    static constexpr int kRowFull = kEpi + 1;                    // query-stationary: the rows' -lse, -delta and exponents landed
    static constexpr int kRowEmpty = kRowFull + 1;               // ... and read (one arrival per elementwise warp)
    static constexpr int kDqFull = kRowEmpty + 1;                // fused kernel: dQ tile of the step complete
    static constexpr int kDqRead = kDqFull + 1;                  // ... and read out (one arrival per warp)
    static constexpr int kPHalf = kDqRead + 1;                   // key-stationary: first half of each P^T slice stored
    static constexpr int kDsHalf = kPHalf + 1;                   // first half of each dS slice stored
    static constexpr int kVFull = kDsHalf + 1;                   // [2] key-stationary: -lse, -delta rows of a step landed
    static constexpr int kVEmpty = kVFull + 2;                   // [2] ... and read (one arrival per elementwise warp)
    // bf16 inputs: tiles converted to fp16 in place (arrivals: one per converting warp)
    static constexpr int kXConv = kVEmpty + 2;                   // stationary tiles (one arrival per elementwise warp)
    static constexpr int kYConv = kXConv + 1;
    static constexpr int kUConv = kYConv + 1;                    // [kUStages] streamed U (warps 18 and 19)
    static constexpr int kWConv = kUConv + kUStages;             // [kWStages] streamed W, key-stationary kernels only
    static constexpr int kBiasFull = kWConv + kWStages;          // PREC = 2: the step's bias tile has landed
    static constexpr int kBiasEmpty = kBiasFull + 1;             // ... and has been read (one arrival per elementwise warp)
    static constexpr int kSums = kBiasEmpty + 1;                 // pairs, MODE 1: the rows' partial sums (elementwise warps)
    static constexpr int kNumBars = kSums + 1;
    // two slots of lse[128] | delta[128]; MODE 1: the rows' lse[128] | delta[128] | exponents[128], pairs: later a partial
    // sum of each row from every warpgroup
    static constexpr int kVecBytes = MODE != 1 ? 2 * 1024 : (PREC ? 128 * 4 * kNWG : 3 * 512);
    static constexpr int kDsBytes = 128 * 128 * 2;               // fused kernel: dS^T tile for the dQ MMA
    static constexpr int kBarBytes = (kNumBars * 8 + 15) / 16 * 16;
    // behind the barriers: TMEM slot, abort flag and wait limit (16 bytes), the answer to a request for a block (16),
    // two BwdItem
    static constexpr int kCtlBytes = 32 + 2 * 48;
    // bytes used from the 1024-aligned base: X, Y, U ring, W ring, [dS], [vectors], barriers, control words, [masks]
    static constexpr int kUsedBytes = (2 + kUStages + kWStages) * kTileBytes + kBiasBytes + (kFused ? kDsBytes : 0) + kVecBytes +
                                      kBarBytes + kCtlBytes + (kMasks ? kMaskBytes : 0);
    static constexpr int kMaxSmem = 232448;                      // 227 KB: the most one CTA can ask for
    static_assert(128 * kNWG + 128 == 32 * tile::kBwdWarps, "thread count and table disagree");
    static_assert(kUsedBytes <= kMaxSmem, "shared-memory plan does not fit");
    // what the launch asks for: room to align the base when it fits (the kernel checks what it got)
    static constexpr int kSmemBytes = kUsedBytes + 1024 <= kMaxSmem ? kUsedBytes + 1024 : kMaxSmem;
};

struct BwdArgs {
    const float* lse2;     // [B*H][nq_pad]  kPShift - lse * log2(e), pairs: -lse; -inf in the padding
    const float* delta;    // [B*H][nq_pad]  -delta, 0 in the padding
    const float* ranges;   // [B*Hkv][2]     max |dO| over the column's query heads, max |V|
    const float* erow;     // [B*H][nq_pad]  row exponents e_i of the fp16 dO copy (row form only)
    float* dq_acc;         // fused kernel: fp32 dQ sums, [B*H][nq_pad/128] tiles of [D/4][128 rows][4]
    const int32_t* kv_len; // optional per-batch key counts
    int32_t* status;
    int B, Nq, Nk, H, Hkv, nq_pad;
    int group;                     // H / Hkv
    int wait_limit_ms;             // limit of a wait for one step (0: the default)
    int cols_per_group;            // CTA order: (batch, head) columns per group, see cta_work()
    int causal;
    int shift;                     // key j is visible to query i iff j <= i + shift
    float scale, scale_log2;
    float score_scale;             // pairs: scale for the scores, with the truncation of their sums given back
    float dp_gain;                 // pairs: the same factor for dP
    // dQ, or dK and dV: 16-byte pieces, element strides
    void* out1; int64_t o1_sb, o1_sn, o1_sh;
    void* out2; int64_t o2_sb, o2_sn, o2_sh;
    uint32_t drop_thr;
    float inv_keep;
    PhiloxKey key;
    DropoutOrigin rng;
    // DROP = 2, the call's keep bits as dropout_bits_kernel lays them out:
    const uint4* bits_q;           // [(b*H + h) * ceil128(Nk)/128 + key tile][nq_pad]: 128 keys of one query row
    const uint32_t* bits_k;        // [((b*H + h) * nq_pad/128 + query tile) * 4 + g][nk_pad]: 32 queries of one key row
    int nk_pad;
    // PREC = 1:
    int d;                         // head size (at most the template's D, a multiple of 8)
    const float* bias;             // optional additive bias, element strides below (0 broadcasts)
    int64_t bias_sb, bias_sn, bias_sh;
    int bias_vec;                  // its rows can be read as float4
    int bias_b, bias_h;            // PREC = 2: whether it has a batch / head dimension
    int ds_vec;                    // rows of d_scores can be written as float4
    int ds_staged;                 // PREC = 2: d_scores leaves by TMA
    float* d_scores;               // optional dense (B, H, Nq, Nk) gradient of the scores (written by MODE 1)
};

__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// ---- number formats of the two operands the threads hand to the MMAs -----------------------------
// P and dS are written to tensor memory as fp16 whatever the input dtype (with bf16 they would carry
// a 2^-9 rounding into dV, dK and dQ at full size; see sm100_ptx.cuh), so both are scaled into
// fp16's range by powers of two that the epilogue takes out again:
//   P'  = P * 2^kPShift                      P <= 1, so P' <= 2^14 and P down to 2^-28 keeps 11 bits
//   dS' = P (dP o Z - delta) * 2^g           g from a bound: |dP o Z - delta| <= 2 D max|dO| max|V| / (1-p)
// and, for bf16 inputs, dO is normalised while it is converted to fp16: dO' = dO * 2^-eO, max|dO'| < 2^15,
// so gradients of any magnitude (bf16 training runs with dO ~ 1e-8) use fp16's range.  max|dO| and max|V|
// are taken per (batch, K/V head) column by the preprocess launch, so a column's result does not depend
// on which other columns the call holds.
constexpr float kPShift = 14.0f;

struct BwdScales {
    float tt_mul;     // dP (as the MMA delivers it) * tt_mul
    float nd_mul;     // the staged -delta vector * nd_mul
    float l_add;      // added to the staged lse vector (key-stationary kernels)
    float ds_mul;     // dS = dS' * ds_mul            (2^-g)
    float acc1_mul;   // dK or dQ  = ACC1 * acc1_mul  (scale * 2^-g)
    float acc2_mul;   // dV        = ACC2 * acc2_mul
    float do_mul;     // inline conversion: dO' = dO * do_mul
};
// smallest k with m < 2^k (0 for m == 0; NaN and infinity count as the largest finite exponent)
__host__ __device__ __forceinline__ int log2_bound_bits(uint32_t bits) {
    bits &= 0x7FFFFFFFu;
    if (bits == 0u) return 0;
    int e = (int)(bits >> 23);
    if (e == 0) return -126;
    if (e > 254) e = 254;
    return e - 127 + 1;
}
__device__ __forceinline__ int log2_bound(float m) { return log2_bound_bits(__float_as_uint(m)); }
__device__ __forceinline__ float pow2i(int e) {
    e = e < -126 ? -126 : (e > 127 ? 127 : e);
    return __uint_as_float((uint32_t)(e + 127) << 23);
}
// How dO reaches the key-stationary kernels' MMAs, which decides where its normalisation sits:
//   kDoAsIs     fp16 inputs: dO is used as it is
//   kDoPairs    bf16 as hi + lo pairs: dO is used as it is, and neither P nor dS needs a scale
//   kDoInline   bf16, converted tile by tile inside the kernel: one factor 2^-e_col for the whole column
//   kDoRowCopy  bf16, converted once by the preprocess launch into an fp16 copy, every row by its own
//               2^-e_i (the column's maximum is not known while the copy is written); the staged vectors
//               hold  lse' = kPShift - lse*log2(e) + e_i  and  -delta * 2^-e_i,  and P carries 2^(e_i - e_col)
// With e_col = (bound of the column's max |dO|) - 15 the constants below are the same in the last two
// forms except for l_add and nd_mul.  The query-stationary kernel multiplies the bf16 dO itself
// (kDoAsIs arithmetic; it undoes e_i in its per-row scalars when the vectors are in the row form).
enum DoForm { kDoAsIs = 0, kDoInline = 1, kDoRowCopy = 2, kDoPairs = 3 };
__device__ __forceinline__ BwdScales make_scales(const float* rng, int D, float inv_keep, float scale, DoForm form) {
    const int k_do = log2_bound(rng[0]), k_v = log2_bound(rng[1]);
    const int e_col = (form == kDoAsIs || form == kDoPairs) ? 0 : k_do - 15;
    // pairs of bf16 have fp32's exponents; elsewhere the factors are whole only within the exponents of normal numbers
    int g = form == kDoPairs ? 0 : 15 - (k_do + k_v + (D > 64 ? 8 : 7) + log2_bound(inv_keep));
    if (form == kDoAsIs) g = g < -112 ? -112 : (g > 126 ? 126 : g);
    BwdScales sc;
    const int up = form == kDoPairs ? 0 : (int)kPShift;       // P' = P * 2^up
    sc.tt_mul = pow2i(g - up + e_col);
    sc.nd_mul = pow2i(g - up + (form == kDoRowCopy ? e_col : 0));
    sc.l_add = form == kDoRowCopy ? (float)(-e_col) : 0.f;
    sc.ds_mul = pow2i(-g);
    sc.acc1_mul = scale * sc.ds_mul;
    sc.acc2_mul = inv_keep * pow2i(e_col - up);
    sc.do_mul = pow2i(-e_col);
    return sc;
}

// Largest magnitude among the eight 16-bit values of a 16-byte piece, folded into a running maximum
// of magnitude bit patterns (two per word; for fp16 and bf16 alike a larger magnitude is a larger
// unsigned pattern).
__device__ __forceinline__ uint32_t absmax16_acc(uint32_t m, const uint4& v) {
    asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.x & 0x7FFF7FFFu));
    asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.y & 0x7FFF7FFFu));
    asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.z & 0x7FFF7FFFu));
    asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.w & 0x7FFF7FFFu));
    return m;
}
// Pairs: the magnitudes of a 16-byte piece that holds an infinity or a NaN are left out.  Such a row's results are no
// numbers whatever the scale; as the column's maximum it pushed the scale of every other row out of range.
template <typename T>
__device__ __forceinline__ uint32_t finite_piece(uint32_t m) {
    constexpr uint32_t inf = std::is_same<T, __half>::value ? 0x7C00u : 0x7F80u;
    return max(m & 0xFFFFu, m >> 16) < inf ? m : 0u;
}
// Which (tile, head, batch) a block of the grid stands for.  The grid is (tiles, heads, batch) and blocks are taken in the
// order of their linear index.  Under a causal mask tiles cost between 1 and `tiles` steps, so the
// order decides how evenly the SMs finish: the (batch, head) columns are taken in groups of
// `cols_per_group`, and within a group all columns' most expensive tile comes first, then the next
// one, ... (longest first).  A group is sized so that its Q, K, V and dO stay in L2 while its CTAs
// run; the cheap tiles that end one group fill the SMs beside the expensive ones that start the next.
struct CtaWork { int tile_rank, head, b; };
__device__ __forceinline__ CtaWork cta_work(int cols_per_group, uint3 block) {
    const int X = (int)gridDim.x, Y = (int)gridDim.y, cols = Y * (int)gridDim.z;
    const int L = (int)block.x + X * ((int)block.y + Y * (int)block.z);
    const int G = cols_per_group < 1 ? 1 : cols_per_group;
    const int grp = L / (G * X), r = L - grp * (G * X);
    const int gcols = (cols - grp * G) < G ? (cols - grp * G) : G;
    const int col = grp * G + r % gcols;
    CtaWork w;
    w.tile_rank = r / gcols;
    w.head = col % Y;
    w.b = col / Y;
    return w;
}

// A block of the grid as the producer leaves it in shared memory for the other roles (twelve words).
struct BwdItem {
    int tile, head_x, b;               // stationary tile; its K/V head (key-stationary) or query head
    int nk;                            // keys the batch entry attends to
    int it0, n_per_head;               // key-stationary: first query tile that sees the tile; steps of a query head
    int n_iter;                        // steps in all; -1: no block any more
    int rot;                           // FUSED: see q_tile_of
    float range[2];                    // max |dO|, max |V| of the column
    int head_kv, pad;
};
static_assert(sizeof(BwdItem) == 48, "kCtlBytes");
template <bool KS, bool FUSED, bool DS>
__device__ __forceinline__ BwdItem make_item(const BwdArgs& a, const CtaWork& cw) {
    BwdItem m;
    m.b = cw.b;
    m.head_x = cw.head;
    m.nk = kv_len_of(a.kv_len, cw.b, a.Nk);
    m.rot = 0;
    if (KS) {
        m.tile = cw.tile_rank;                        // key tile: the first one sees the most query tiles
        m.head_kv = cw.head;
        // first query tile that sees this key tile: query i sees key j iff j <= i + shift
        m.it0 = a.causal ? (m.tile * kTile > a.shift ? (m.tile * kTile - a.shift) / kTile : 0) : 0;
        const int nq_tiles = (a.Nq + kTile - 1) / kTile;
        m.n_per_head = nq_tiles > m.it0 ? nq_tiles - m.it0 : 0;
        if (m.tile * kTile >= m.nk) m.n_per_head = 0;   // a tile of padding keys: dK = dV = 0
        m.n_iter = m.n_per_head * a.group;
        // The fused kernel without a causal mask starts each key tile's walk at a different query tile, so that the CTAs
        // of one head, which run at the same time, add to different dQ tiles (under a causal mask the walks are
        // staggered already).
        if (FUSED && !a.causal && m.n_per_head > 0) m.rot = m.tile % m.n_per_head;
    } else {
        m.tile = a.causal ? (int)gridDim.x - 1 - cw.tile_rank : cw.tile_rank;     // query tile, heavy first
        m.head_kv = cw.head / a.group;
        m.it0 = 0;
        int kv_end = m.nk;
        if (a.causal && m.tile * kTile + kTile + a.shift < kv_end) kv_end = m.tile * kTile + kTile + a.shift;
        m.n_per_head = kv_end > 0 ? (kv_end + kTile - 1) / kTile : 0;
        // d(loss)/d(scores) wanted: the steps are walked twice (comment at `sum_p2` below)
        m.n_iter = DS ? 2 * m.n_per_head : m.n_per_head;
    }
    return m;
}

// MODE 0: dK, dV (key-stationary).  MODE 1: dQ (query-stationary).
// INLINE (bf16 inputs only): the streamed tiles arrive as bf16 and warps 18 and 19 convert them;
// otherwise bf16 calls stream the fp16 copies the preprocess launch (Q, dO) and the dK/dV kernel (K:
// map_aux, a by-product of its stationary tile) have written to the workspace.
// DS (pairs, MODE 1): the call wants d(loss)/d(scores).  An instance of its own: as branches its code cost the kernel of
// calls that do not want it 13 of 66 us (B4 N1024 H16 D96 causal).  Two walks over the keys take 95 us where one took 71
// (B8 N512 H12 D64 bf16); see `sum_p2` for what they give.
template <int D, bool BF16, int MODE, int NWG, int DROP, bool INLINE, int PREC, bool DS>
__global__ void __launch_bounds__(128 * NWG + kExtraThreads, 1)
bwd_sm100_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                 const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_out1, const __grid_constant__ CUtensorMap map_out2,
                 const __grid_constant__ CUtensorMap map_aux, const __grid_constant__ CUtensorMap map_bias,
                 const __grid_constant__ CUtensorMap map_ds, const BwdArgs a) {
    using Cfg = BwdCfg<D, MODE, DROP, PREC>;
    constexpr bool KS = (MODE != 1);        // key-stationary: K, V stay, query tiles stream
    constexpr bool FUSED = (MODE == 2);     // key-stationary and dQ too
    constexpr bool CONV = BF16 && PREC == 0;    // every MMA runs f16 x f16: bf16 tiles are converted
    constexpr bool P_BF16 = BF16 && PREC != 0;  // ... except that pairs of bf16 need no conversion
    static_assert(PREC == 0 || (MODE != 2 && !INLINE), "the pair instances are the two-pass form");
    constexpr bool STREAM_CONV = CONV && INLINE;             // ... the streamed ones by warps 18 and 19
    constexpr bool XY_CONV = CONV && (KS || INLINE);         // ... the stationary ones (X; key-stationary also Y), too
    constexpr bool ROWFORM = CONV && !INLINE;                // staged vectors are in the row form (see DoForm)
    constexpr bool K_COPY = ROWFORM && MODE == 0;            // this kernel writes the fp16 copy of K
    constexpr bool ROW_MAX = PREC != 0 && !BF16 && MODE == 1;   // the threads read Y, too
    static_assert(BF16 || !INLINE, "inline conversion is a bf16 variant");
    constexpr int UST = Cfg::kUStages, WST = Cfg::kWStages;
    constexpr int TILE = Cfg::kTileBytes;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sX = smem;
    uint8_t* sY = sX + TILE;
    uint8_t* sU = sY + TILE;                        // U ring
    uint8_t* sW = sU + UST * TILE;                  // W ring
    uint8_t* sBias = sW + WST * TILE;               // PREC = 2
    uint8_t* sDs = sBias + Cfg::kBiasBytes;         // fused kernel only
    float* sVec = (float*)(sDs + (FUSED ? Cfg::kDsBytes : 0));      // key-stationary: 2 x (lse[128] | delta[128]); see kVecBytes
    uint64_t* bars = (uint64_t*)((uint8_t*)sVec + Cfg::kVecBytes);
    uint32_t* tmem_slot = (uint32_t*)((uint8_t*)bars + Cfg::kBarBytes);
    volatile uint32_t* abort_flag = (volatile uint32_t*)(tmem_slot + 1);
    uint32_t* clc_answer = tmem_slot + 4;
    volatile BwdItem* sched = (volatile BwdItem*)(tmem_slot + 8);              // [2]: block k of this CTA in slot k & 1
    uint16_t* sMask = (uint16_t*)((uint8_t*)bars + Cfg::kBarBytes + Cfg::kCtlBytes);    // present with dropout only
    {
        // the launch may have had no room for a full kilobyte of alignment slack
        uint32_t dyn;
        asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if ((uint32_t)(smem - smem_raw) + (uint32_t)Cfg::kUsedBytes > dyn) {
            if (threadIdx.x == 0) report_status(a.status, 8);
            return;
        }
    }

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // query-stationary: key tile of step `it`
    auto k_tile_of = [&](int n_per_head, int it) { return DS && it >= n_per_head ? it - n_per_head : it; };
    // Key-stationary kernels: query tile of a step, qi = its index within its query head (each role keeps qi and the head
    // count as running counters: a division per step and warp is a visible share of the issue slots).
    auto q_tile_of = [&](int it0, int n_per_head, int rot, int qi) {
        int t = qi + rot;
        if (t >= n_per_head) t -= n_per_head;
        return it0 + t;
    };

    constexpr int kMmaWarp = 4 * NWG, kTmaWarp = 4 * NWG + 1;
    constexpr int CPT = kTile / NWG;                    // columns of T1/T2 one elementwise thread owns
    constexpr int kAllThreads = 128 * NWG + kExtraThreads;
    if (warp == kTmaWarp) {
        // the producer's warp sets the barriers up, so that the first loads need not wait for the other warps
        constexpr uint32_t kReaders = 4u * NWG + 2u + ((STREAM_CONV || PREC == 2) ? 1u : 0u);
        for (int i = lane; i < Cfg::kNumBars; i += 32) {
            const bool wide = (i == Cfg::kPReady || i == Cfg::kDsReady || i == Cfg::kMask || i == Cfg::kEpi || i == Cfg::kRowEmpty ||
                               i == Cfg::kXConv || i == Cfg::kYConv ||
                               i == Cfg::kDqRead || i == Cfg::kPHalf || i == Cfg::kDsHalf ||
                               i == Cfg::kVEmpty || i == Cfg::kVEmpty + 1 || i >= Cfg::kBiasEmpty);
            const bool conv2 = i >= Cfg::kUConv && i < Cfg::kBiasFull;          // the two converting warps
            uint32_t count = wide ? 4u * NWG : (conv2 ? 2u : 1u);    // one arrival per elementwise warp
            if (i == Cfg::kSchedEmpty || i == Cfg::kSchedEmpty + 1) count = kReaders;
            if (i == Cfg::kXEmpty && K_COPY) count = 2u;              // the MMAs and the copy of K
            if (i == Cfg::kYEmpty && ROW_MAX) count = 1u + 4u * NWG;
            mbar_init(&bars[i], count);
        }
        if (lane == 0) wait_control_init(abort_flag, a.wait_limit_ms);
        fence_mbar_init();
        __syncwarp();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == kTmaWarp) {
        asm volatile("barrier.cta.arrive 1, %0;" ::"n"(kAllThreads) : "memory");
    } else {
        tc_fence_before_sync();
        asm volatile("barrier.cta.sync 1, %0;" ::"n"(kAllThreads) : "memory");
        tc_fence_after_sync();
    }
    if (MODE == 0) {
        // The preprocess launch's vectors and copies: what stands above runs beside its end (3 us of a step).
        grid_dependency_wait();
        // The dQ kernel reads nothing the dK/dV kernel writes: it may take the SMs this grid's last wave
        // leaves idle (it is launched serialized behind this grid, and waits for it only before it ends).
        grid_launch_dependents();
    }
    const uint32_t tmem = *tmem_slot;
    const uint32_t tT1 = tmem, tT2 = tmem + 128u, tAcc1 = tmem + 256u, tAcc2 = tmem + 384u;
    const uint32_t tDq = tmem + 448u;                   // fused kernel (D = 64 only): the per-step dQ tile
    constexpr DoForm kForm = P_BF16 ? kDoPairs : (!(CONV && KS) ? kDoAsIs : (INLINE ? kDoInline : kDoRowCopy));

    // Persistent: a CTA goes on to a further block of the grid, which it takes from the blocks not yet launched
    // (clusterlaunchcontrol), so the order above and its balance stay what the hardware's dispatch gives, and the streamed
    // tiles, the rings' and barriers' phases and tensor memory carry on.  As a CTA per block, the start (barriers, tensor
    // memory, the first loads), the end and the gap between two CTAs cost 13900 cycles a block of the dK/dV kernel and
    // 11000 of the dQ kernel at D = 128 bf16, 8900 and 8700 at D = 64 fp16, next to 2700, 1570, 2350 and 1460 a step.
    // The producer asks for the next block and leaves it in one of two slots; k counts a role's blocks.  A role that is
    // done with a slot arrives on its barrier (the elementwise warps at a block's end: they read the slot again instead of
    // holding it in registers).
    auto item_there = [&](int k) { return mbar_wait(&bars[Cfg::kSchedFull + (k & 1)], (uint32_t)(k >> 1) & 1u, abort_flag); };

    // Registers: without dropout the launch allocation of 96 per thread is enough for all but a few words (-Xptxas -v: 8
    // bytes stored and 20 loaded in the bf16 dK/dV instances, which is 0.1 % of their instructions under ncu; up to 80 and
    // 88 in those that write d(loss)/d(scores), 32 and 44 in the one-kernel form), and moving
    // registers from the MMA / TMA warps to the elementwise ones (104 / 64, 104 / 40) made one side or the
    // other spill and measured the same or slower.  The dK/dV kernel's dropout instances spill in the
    // elementwise loop: they take 104 and leave 64 to the other warpgroup (1.272 -> 1.216 ms at
    // B32 H16 N2048 D64; the one-kernel backward got slower with the same split, 1.439 -> 1.466, and keeps 96).  With 104
    // it is 17 local loads and 12 stores a step and warp, 5 % of the instructions (ncu, B4 N2048 H16 D64 causal).
    constexpr bool kMoveRegs = DROP != 0 && MODE == 0 && !INLINE;
    // The pool is what the CTA was launched with (96 per thread): a split that asks for more makes
    // setmaxnreg.inc wait for ever (112 / 40 did: 62464 > 61440).
    constexpr int kRegsElementwiseMoved = 104, kRegsOtherMoved = 64, kRegsLaunch = 96;
    static_assert(128 * NWG * kRegsElementwiseMoved + kExtraThreads * kRegsOtherMoved <= (128 * NWG + kExtraThreads) * kRegsLaunch,
                  "register split exceeds the launch allocation");
    if (warp >= kMmaWarp) {
      if constexpr (kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOtherMoved));
      if (warp == kTmaWarp) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            prefetch_tensormap(&map_x); prefetch_tensormap(&map_u);
            int u_issued = 0, w_issued = 0, v_issued = 0, r_issued = 0, items = 0, asked = 0;     // items: blocks with steps
            int us = 0, ws = 0;                      // ring slots of this step
            uint32_t uph = 0, wph = 0;               // how often each ring has wrapped (parity)
            int xy_issued[2] = {0, 0};
            bool ok = true;
            CtaWork w = cta_work(a.cols_per_group, blockIdx);
            BwdItem m = make_item<KS, FUSED, DS>(a, w);
            auto publish = [&](int k) {
                const int slot = k & 1;
                float2 rg = make_float2(0.f, 0.f);
                if (m.n_iter >= 0) rg = *reinterpret_cast<const float2*>(a.ranges + 2 * ((int64_t)m.b * a.Hkv + m.head_kv));
                ok = mbar_wait(&bars[Cfg::kSchedEmpty + slot], ((uint32_t)(k >> 1) & 1u) ^ 1u, abort_flag);
                if (!ok) return;
                volatile BwdItem* d = sched + slot;
                d->tile = m.tile; d->head_x = m.head_x; d->b = m.b; d->nk = m.nk; d->it0 = m.it0; d->n_per_head = m.n_per_head;
                d->n_iter = m.n_iter; d->rot = m.rot; d->range[0] = rg.x; d->range[1] = rg.y; d->head_kv = m.head_kv;
                mbar_arrive(&bars[Cfg::kSchedFull + slot]);
            };
            for (int k = 0; ok; ++k) {
                bool published = k > 0;              // (the first block's loads go out first)
                auto load_xy = [&](int y) {
                    ok = mbar_wait(&bars[Cfg::kXEmpty + y], ((uint32_t)items & 1u) ^ 1u, abort_flag);
                    if (!ok) return;
                    mbar_expect_tx(&bars[Cfg::kXFull + y], TILE);
#pragma unroll
                    for (int bx = 0; bx < Cfg::kNBox; ++bx)
                        tma_load_4d(sX + y * TILE + bx * kBoxBytes, y ? &map_y : &map_x, &bars[Cfg::kXFull + y], bx * 64, m.head_x, m.tile * kTile, m.b);
                    ++xy_issued[y];
                };
                int qi = 0, hg = 0;
                for (int it = 0; it < m.n_iter; ++it) {
                    int head_u, row_u;
                    if (KS) { head_u = m.head_x * a.group + hg; row_u = q_tile_of(m.it0, m.n_per_head, m.rot, qi) * kTile; }
                    else    { head_u = m.head_kv; row_u = k_tile_of(m.n_per_head, it) * kTile; }
                    ok = mbar_wait(&bars[Cfg::kUEmpty + us], (uph & 1u) ^ 1u, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&bars[Cfg::kUFull + us], TILE);
#pragma unroll
                    for (int bx = 0; bx < Cfg::kNBox; ++bx)
                        tma_load_4d(sU + us * TILE + bx * kBoxBytes, &map_u, &bars[Cfg::kUFull + us], bx * 64, head_u, row_u, m.b);
                    ++u_issued;
                    if (it == 0) { load_xy(0); if (!ok) break; }
                    ok = mbar_wait(&bars[Cfg::kWEmpty + ws], (wph & 1u) ^ 1u, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&bars[Cfg::kWFull + ws], TILE);
#pragma unroll
                    for (int bx = 0; bx < Cfg::kNBox; ++bx)
                        tma_load_4d(sW + ws * TILE + bx * kBoxBytes, &map_w, &bars[Cfg::kWFull + ws], bx * 64, head_u, row_u, m.b);
                    ++w_issued;
                    if (KS) {
                        // the step's -lse*log2(e) and -delta rows: a two-slot ring of their own
                        const int vs = v_issued & 1;
                        ok = mbar_wait(&bars[Cfg::kVEmpty + vs], ((uint32_t)(v_issued >> 1) & 1u) ^ 1u, abort_flag);
                        if (!ok) break;
                        const int64_t off = ((int64_t)m.b * a.H + head_u) * a.nq_pad + row_u;
                        mbar_expect_tx(&bars[Cfg::kVFull + vs], 1024);
                        bulk_load_1d(sVec + vs * 256, a.lse2 + off, 512, &bars[Cfg::kVFull + vs]);
                        bulk_load_1d(sVec + vs * 256 + 128, a.delta + off, 512, &bars[Cfg::kVFull + vs]);
                        ++v_issued;
                    } else if (it == 0) {
                        // the stationary rows' own: read by the threads when the block begins
                        ok = mbar_wait(&bars[Cfg::kRowEmpty], ((uint32_t)items & 1u) ^ 1u, abort_flag);
                        if (!ok) break;
                        const int64_t off = ((int64_t)m.b * a.H + m.head_x) * a.nq_pad + m.tile * kTile;
                        mbar_expect_tx(&bars[Cfg::kRowFull], ROWFORM ? 1536 : 1024);
                        bulk_load_1d(sVec, a.lse2 + off, 512, &bars[Cfg::kRowFull]);
                        bulk_load_1d(sVec + 128, a.delta + off, 512, &bars[Cfg::kRowFull]);
                        if (ROWFORM) bulk_load_1d(sVec + 256, a.erow + off, 512, &bars[Cfg::kRowFull]);
                        ++r_issued;
                    }
                    if (it == 0) { load_xy(1); if (!ok) break; }
                    if (++us == UST) { us = 0; ++uph; }
                    if (++ws == WST) { ws = 0; ++wph; }
                    if (++qi == m.n_per_head) { qi = 0; ++hg; }
                    if (!published) { publish(k); published = true; if (!ok) break; }
                    // a request two steps before the last one: its answer is there in time, and the block is
                    // not taken from a CTA that would have come to it sooner
                    if (it + 3 >= m.n_iter && asked == k) { clc_request(clc_answer, &bars[Cfg::kClc]); ++asked; }
                }
                if (ok && !published) publish(k);
                if (!ok) break;
                if (m.n_iter > 0) ++items;
                if (asked == k) { clc_request(clc_answer, &bars[Cfg::kClc]); ++asked; }
                ok = mbar_wait(&bars[Cfg::kClc], (uint32_t)k & 1u, abort_flag);
                if (!ok) break;
                uint3 block;
                const bool another = clc_answer_block(clc_answer, block);
                fence_proxy_async_smem();            // read before the next answer is written
                if (another) m = make_item<KS, FUSED, DS>(a, cta_work(a.cols_per_group, block));
                else m.n_iter = -1;
                publish(k + 1);
                if (!another) break;
            }
            if (!ok) {
                // unwinding: let copies already issued land before shared memory is given up
                auto landed = [&](int bar, int n) {
                    for (int spin = 0; spin < 4096 && n > 0 && !mbar_try_wait(&bars[bar], (uint32_t)(n - 1) & 1u); ++spin) {}
                };
                for (int st = 0; st < UST; ++st) landed(Cfg::kUFull + st, (u_issued + UST - 1 - st) / UST);
                for (int st = 0; st < WST; ++st) landed(Cfg::kWFull + st, (w_issued + WST - 1 - st) / WST);
                for (int st = 0; st < 2; ++st) landed(Cfg::kVFull + st, (v_issued + 1 - st) / 2);
                for (int y = 0; y < 2; ++y) landed(Cfg::kXFull + y, xy_issued[y]);
                landed(Cfg::kRowFull, r_issued);
                landed(Cfg::kClc, asked);
            }
        }
        __syncwarp();
      } else if (warp == kMmaWarp) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            // operand formats: converted tiles, P and dS are fp16; the query-stationary kernel's dP keeps
            // its two bf16 tiles (dO_i, V_j) as they are
            constexpr bool T1_BF16 = BF16 && !CONV, T2_BF16 = BF16 && !(CONV && KS);
            constexpr uint32_t idesc_t1 = make_idesc_f16(T1_BF16, T1_BF16, kTile, kTile, false, false);
            constexpr uint32_t idesc_t2 = make_idesc_f16(T2_BF16, T2_BF16, kTile, kTile, false, false);
            const uint32_t idesc_acc = PREC ? make_idesc_f16(P_BF16, P_BF16, kTile, (a.d + 15) & ~15, false, true)
                                            : make_idesc_f16(false, false, kTile, D, false, true);
            constexpr int kUReady = STREAM_CONV ? Cfg::kUConv : Cfg::kUFull;
            constexpr int kWReady = (STREAM_CONV && KS) ? Cfg::kWConv : Cfg::kWFull;
            constexpr int kXReady = XY_CONV ? Cfg::kXConv : Cfg::kXFull;
            constexpr int kYReady = (XY_CONV && KS) ? Cfg::kYConv : Cfg::kYFull;
            const uint32_t sX_u = smem_u32(sX), sY_u = smem_u32(sY), sU_u = smem_u32(sU), sW_u = smem_u32(sW);

            // Descriptors differ only in the 16-byte-granular start address held in their low
            // bits: build the two kinds once and add offsets in the issue loops, which keeps the
            // single issuing thread's instruction count per MMA small.
            const uint64_t dk_major = make_smem_desc_sw128(0, 0, 1024);            // K-major operand
            const uint64_t dmn_major = make_smem_desc_sw128(0, kBoxBytes, 1024);   // MN-major operand
            auto issue_t = [&](uint32_t d_tmem, uint32_t stat_u, uint32_t strm_u, uint32_t idesc_t) {
                const uint64_t a0 = dk_major + (uint64_t)(stat_u >> 4), b0 = dk_major + (uint64_t)(strm_u >> 4);
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const uint32_t off = ((uint32_t)(kk >> 2) * kBoxBytes + (uint32_t)(kk & 3) * 32u) >> 4;
                    if (PREC == 0 || kk * 16 < a.d) mma_ss_f16(d_tmem, a0 + off, b0 + off, idesc_t, kk > 0);
                }
            };
            // acc (+)= A[TMEM] * B[smem tile, MN-major], restricted to the first (hf = 0) or second 16 columns of
            // every warpgroup's slice: K-steps kk = hf, hf + 2, hf + 4, hf + 6.  A holds 16-bit pairs: the group
            // that owns columns [g*CPT, (g+1)*CPT) of T wrote its CPT values packed into columns
            // [g*CPT, g*CPT + CPT/2); with pairs their low parts follow in [g*CPT + CPT/2, (g+1)*CPT).
            auto issue_acc_half = [&](uint32_t d_tmem, uint32_t a_tmem, uint32_t strm_u, bool acc, int hf) {
                static_assert(CPT == 32, "one K-step of 16 per half slice");
                const uint64_t b0 = dmn_major + (uint64_t)(strm_u >> 4);
#pragma unroll
                for (int q = 0; q < kTile / 32; ++q) {
                    const int kk = 2 * q + hf;
                    const uint32_t a_col = (uint32_t)q * CPT + (uint32_t)hf * 8u;
                    mma_ts_f16(d_tmem, a_tmem + a_col, b0 + (uint64_t)((kk * 2048) >> 4), idesc_acc,
                               (acc || hf > 0 || q > 0) ? 1u : 0u);
                    if (PREC) mma_ts_f16(d_tmem, a_tmem + a_col + CPT / 2, b0 + (uint64_t)((kk * 2048) >> 4), idesc_acc, 1u);
                }
            };

            // fused kernel: the step's dQ tile (fresh accumulation) from two shared-memory operands
            constexpr uint32_t idesc_dq = make_idesc_f16(false, false, kTile, D, true, true);
            const uint32_t sDs_u = smem_u32(sDs);
            auto issue_dq = [&]() {
                const uint64_t a0 = dmn_major + (uint64_t)(sDs_u >> 4), b0 = dmn_major + (uint64_t)(sX_u >> 4);
#pragma unroll
                for (int kk = 0; kk < kTile / 16; ++kk)
                    mma_ss_f16(tDq, a0 + (uint64_t)((kk * 2048) >> 4), b0 + (uint64_t)((kk * 2048) >> 4), idesc_dq,
                               kk > 0);
            };

            // A block's first S and dP are issued behind the last MMAs of the block before it; its accumulators are first
            // written behind a hand-off that the threads make when they have read those of the block before.
            // The loop over the steps holds nothing but a step: this thread is what a step waits for, and with a block's start
            // folded into the loop the dQ kernel took 154 us for 128 steps instead of 138 (one head, N 16384, D 128), the
            // other one 225 instead of 218.
            bool ok = true;
            int blocks = 0, items = 0, g = 0;        // blocks, blocks with steps, steps so far
            int us = 0, ws = 0;                      // ring slots of this step's U and W
            uint32_t uph = 0, wph = 0;               // wrap counts (parity of the slots' phases)
            for (;;) {
                // (blocks without steps one at a time: the threads are done with a block's slot when they have ended the block,
                // and there are two slots)
                ok = item_there(blocks);
                if (!ok) break;
                const int n_iter = sched[blocks & 1].n_iter;
                [[maybe_unused]] const int sum_steps = DS ? sched[blocks & 1].n_per_head : 0;
                mbar_arrive(&bars[Cfg::kSchedEmpty + (blocks & 1)]);
                ++blocks;
                if (n_iter < 0) break;
                if (n_iter == 0) continue;
                ok = mbar_wait(&bars[kUReady + us], uph & 1u, abort_flag);
                if (ok) ok = mbar_wait(&bars[kXReady], (uint32_t)items & 1u, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                issue_t(tT1, sX_u, sU_u + us * TILE, idesc_t1);
                mma_commit(&bars[Cfg::kT1Full]);
                if (n_iter == 1 && !FUSED) mma_commit(&bars[Cfg::kXEmpty]);
                ok = mbar_wait(&bars[kWReady + ws], wph & 1u, abort_flag);
                if (ok) ok = mbar_wait(&bars[kYReady], (uint32_t)items & 1u, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                issue_t((!KS && (g & 1)) ? tAcc2 : tT2, sY_u, sW_u + ws * TILE, idesc_t2);
                mma_commit(&bars[(!KS && (g & 1)) ? Cfg::kT1Full + 1 : Cfg::kT2Full]);
                if (!KS) mma_commit(&bars[Cfg::kWEmpty + ws]);               // MODE 1: V_j is read by dP(j) only
                if (n_iter == 1) mma_commit(&bars[Cfg::kYEmpty]);
                for (int it = 0; it < n_iter; ++it, ++g) {
                    int nus = us + 1, nws = ws + 1;      // slots of the next step
                    uint32_t nuph = uph, nwph = wph;
                    if (nus == UST) { nus = 0; ++nuph; }
                    if (nws == WST) { nws = 0; ++nwph; }
                    const uint32_t cur_u = sU_u + us * TILE, nxt_u = sU_u + nus * TILE;
                    const uint32_t cur_w = sW_u + ws * TILE, nxt_w = sW_u + nws * TILE;
                    const bool more = it + 1 < n_iter, ends = it + 2 == n_iter;      // ends: the next step is the block's last
                    if (more) { ok = mbar_wait(&bars[kUReady + nus], nuph & 1u, abort_flag); if (!ok) break; }
                    if (KS) {
                        ok = mbar_wait(&bars[Cfg::kPHalf], (uint32_t)g & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_acc_half(tAcc2, tT1, cur_w, it > 0, 0);                // dV += (P o Z)^T dO, first halves
                        ok = mbar_wait(&bars[Cfg::kPReady], (uint32_t)g & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_acc_half(tAcc2, tT1, cur_w, it > 0, 1);
                        if (more) {
                            mma_commit(&bars[Cfg::kWEmpty + ws]);                    // dO_i: dP^T(i) earlier, dV(i) last
                            issue_t(tT1, sX_u, nxt_u, idesc_t1);
                            mma_commit(&bars[Cfg::kT1Full]);
                            if (ends && !FUSED) mma_commit(&bars[Cfg::kXEmpty]);
                        }
                    } else if (more) {
                        // dQ needs no second accumulator, and P never goes back to tensor memory here: S has one
                        // buffer, free again as soon as the threads hold S(it) in registers, and dP / dS have
                        // two (T2 and the columns a second accumulator would take).  S(it+1) and dP(it+1) are
                        // both issued before this thread waits for dS(it), so the threads find their next
                        // inputs ready; with one dP buffer, dP(it+1) could only follow dQ(it), and
                        // dS -> dQ -> dP -> dS was the loop that set the step time.
                        ok = mbar_wait(&bars[Cfg::kPReady], (uint32_t)g & 1u, abort_flag);     // S(it) is in registers
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_t(tT1, sX_u, nxt_u, idesc_t1);
                        mma_commit(&bars[Cfg::kT1Full]);
                        ok = mbar_wait(&bars[kWReady + nws], nwph & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        // the buffer of step it+1 held dS(it-1), which dQ(it-1) read: issued before, in order
                        issue_t(((g + 1) & 1) ? tAcc2 : tT2, sY_u, nxt_w, idesc_t2);
                        mma_commit(&bars[((g + 1) & 1) ? Cfg::kT1Full + 1 : Cfg::kT2Full]);
                        mma_commit(&bars[Cfg::kWEmpty + nws]);
                        if (ends) { mma_commit(&bars[Cfg::kXEmpty]); mma_commit(&bars[Cfg::kYEmpty]); }
                    }
                    // query-stationary: a barrier pair per dP / dS buffer (phase = uses of that buffer), which
                    // the threads cannot lap: dS(it+2) needs dP(it+2), issued after these waits
                    const int b_half = (!KS && (g & 1)) ? Cfg::kPHalf : Cfg::kDsHalf;
                    const int b_ready = (!KS && (g & 1)) ? Cfg::kDqRead : Cfg::kDsReady;
                    const uint32_t ds_par = KS ? ((uint32_t)g & 1u) : ((uint32_t)(g >> 1) & 1u);
                    const uint32_t tDs = (!KS && (g & 1)) ? tAcc2 : tT2;
                    ok = mbar_wait(&bars[b_half], ds_par, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const bool acc = !DS || it >= sum_steps;                       // (no dS in the steps that only sum)
                    if (acc) issue_acc_half(tAcc1, tDs, cur_u, it > sum_steps, 0);   // dK += dS^T Q  /  dQ += dS K
                    ok = mbar_wait(&bars[b_ready], ds_par, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (acc) issue_acc_half(tAcc1, tDs, cur_u, it > sum_steps, 1);
                    // last reader of U(it); a block's last U and W tiles' places take its results first
                    mma_commit(&bars[more ? Cfg::kUEmpty + us : Cfg::kAccDone]);
                    if (FUSED) {
                        // dQ tile of this step = dS K_j: A is the dS^T tile the threads left in shared memory,
                        // read MN-major (M = queries), B is the stationary K tile read MN-major (N = D).  Only the previous
                        // tile's read-out has to precede (issuing dP^T(it+1) ahead of this MMA measured slower)
                        if (g > 0) {
                            ok = mbar_wait(&bars[Cfg::kDqRead], (uint32_t)(g - 1) & 1u, abort_flag);
                            if (!ok) break;
                            tc_fence_after_sync();
                        }
                        issue_dq();
                        mma_commit(&bars[Cfg::kDqFull]);
                        if (!more) mma_commit(&bars[Cfg::kXEmpty]);
                    }
                    if (KS && more) {
                        ok = mbar_wait(&bars[kWReady + nws], nwph & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_t(tT2, sY_u, nxt_w, idesc_t2);
                        mma_commit(&bars[Cfg::kT2Full]);
                        if (ends) mma_commit(&bars[Cfg::kYEmpty]);
                    }
                    us = nus; uph = nuph; ws = nws; wph = nwph;
                }
                if (!ok) break;
                // query-stationary: the next block's S overwrites the last one's, which has to be in registers
                if (!KS) ok = mbar_wait(&bars[Cfg::kPReady], (uint32_t)(g - 1) & 1u, abort_flag);
                if (!ok) break;
                ++items;
            }
        }
        __syncwarp();
      } else if (warp == kTmaWarp + 2 || STREAM_CONV) {
        // ---------------------------------------------------------------- warp 19: TMA stores (K's copy, the results)
        // INLINE, with warp 18: the streamed tiles bf16 -> fp16, between their arrival (U_full, W_full) and their first
        // reader (the MMAs wait for U_conv, W_conv), dO tiles normalised on the way.
        const int ct = (warp - kTmaWarp - 1) * 32 + lane;
        const bool stores = warp == kTmaWarp + 2 && lane == 0;
        constexpr uint32_t kIdleNs = 200;          // (looking all the time it slowed every step by a tenth)
        int us = 0, ws = 0, items = 0, steps = 0;
        uint32_t uph = 0, wph = 0;
        bool ok = true;
        auto convert = [&](int full, int conv, uint32_t parity, uint8_t* tile, bool scaled, float mul) {
            ok = mbar_wait(&bars[full], parity & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            if (scaled) convert_tile_bf16_to_f16<true>(tile, TILE, ct, 64, mul);
            else        convert_tile_bf16_to_f16<false>(tile, TILE, ct, 64, 1.f);
            fence_proxy_async_smem();
            mbar_arrive_warp(&bars[conv]);
        };
        for (int k = 0; ; ++k) {
            ok = ok && mbar_wait(&bars[Cfg::kSchedFull + (k & 1)], (uint32_t)(k >> 1) & 1u, abort_flag, STREAM_CONV ? 0u : kIdleNs);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const volatile BwdItem* m = sched + (k & 1);
            const int n_iter = m->n_iter, row0 = m->tile * kTile, head = m->head_x, b = m->b;
            const float range[2] = {m->range[0], m->range[1]};
            mbar_arrive_warp(&bars[Cfg::kSchedEmpty + (k & 1)]);
            if (n_iter < 0) break;
            if (n_iter == 0) continue;
            if (K_COPY && stores && mbar_wait(&bars[Cfg::kXConv], (uint32_t)items & 1u, abort_flag, kIdleNs)) {
                // the fp16 K tile is what the dQ kernel streams: keep a copy (rows beyond Nk are clipped)
#pragma unroll
                for (int bx = 0; bx < Cfg::kNBox; ++bx)
                    tma_store_4d(&map_aux, sX + bx * kBoxBytes, bx * 64, head, row0, b);
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(&bars[Cfg::kXEmpty]);
            }
            __syncwarp();
            if (STREAM_CONV) {
                const float do_mul = make_scales(range, D, a.inv_keep, a.scale, kForm).do_mul;
                for (int it = 0; it < n_iter && ok; ++it) {
                    convert(Cfg::kUFull + us, Cfg::kUConv + us, uph, sU + us * TILE, false, 1.f);
                    if (KS && ok) convert(Cfg::kWFull + ws, Cfg::kWConv + ws, wph, sW + ws * TILE, true, do_mul);
                    if (++us == UST) { us = 0; ++uph; }
                    if (++ws == WST) { ws = 0; ++wph; }
                }
                if (!ok) break;
            }
            steps += n_iter;
            // (all the block's steps lie in this wait, beside the next one's start)
            if (stores && mbar_wait(&bars[Cfg::kEpi], (uint32_t)items & 1u, abort_flag, kIdleNs, (uint32_t)n_iter + 1u)) {
                const int su = (steps - 1) % UST, sw = (steps - 1) % WST;
#pragma unroll
                for (int bx = 0; bx < Cfg::kNBox; ++bx) {
                    tma_store_4d(&map_out1, sU + su * TILE + bx * kBoxBytes, bx * 64, head, row0, b);
                    if (KS) tma_store_4d(&map_out2, sW + sw * TILE + bx * kBoxBytes, bx * 64, head, row0, b);
                }
                tma_store_commit();
                tma_store_wait_read<0>();          // (the writes complete on their own)
                mbar_arrive(&bars[Cfg::kUEmpty + su]);
                if (KS) mbar_arrive(&bars[Cfg::kWEmpty + sw]);
            }
            __syncwarp();
            ++items;
        }
      } else if (PREC == 2 && warp == kTmaWarp + 1) {
        // ---------------------------------------------------------------- warp 18: the steps' bias tiles
        if (elect_one()) {
            int done = 0;                        // tiles loaded so far
            bool ok = true;
            for (int k = 0; ok; ++k) {
                ok = item_there(k);
                if (!ok) break;
                const volatile BwdItem* m = sched + (k & 1);
                const int n_iter = m->n_iter, n_per_head = m->n_per_head, it0 = m->it0, head_x = m->head_x, tile = m->tile, b = m->b;
                mbar_arrive(&bars[Cfg::kSchedEmpty + (k & 1)]);
                if (n_iter < 0) break;
                const int sum_steps = DS ? n_per_head : 0;
                int qi = 0, hg = 0;
                // dQ kernel: the threads leave d(loss)/d(scores) of a step in the place of its bias tile
                auto store_ds = [&](int it) {
                    const int k_col = k_tile_of(n_per_head, it) * kTile;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (k_col + 32 * c < a.Nk) tma_store_4d(&map_ds, sBias + c * kBoxBytes, k_col + 32 * c, head_x, tile * kTile, b);
                    tma_store_commit();
                    tma_store_wait_read<0>();
                };
                for (int it = 0; it < n_iter; ++it) {
                    const int head = KS ? head_x * a.group + hg : head_x;
                    const int q_row = (KS ? q_tile_of(it0, n_per_head, 0, qi) : tile) * kTile;
                    const int k_col = (KS ? tile : k_tile_of(n_per_head, it)) * kTile;
                    ok = mbar_wait(&bars[Cfg::kBiasEmpty], ((uint32_t)done & 1u) ^ 1u, abort_flag);
                    if (!ok) break;
                    if (DS && a.ds_staged && it > sum_steps) store_ds(it - 1);
                    mbar_expect_tx(&bars[Cfg::kBiasFull], 4 * kBoxBytes);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        tma_load_4d(sBias + c * kBoxBytes, &map_bias, &bars[Cfg::kBiasFull], k_col + 32 * c, a.bias_h ? head : 0, q_row,
                                    a.bias_b ? b : 0);
                    ++done;
                    if (++qi == n_per_head) { qi = 0; ++hg; }
                }
                if (DS && a.ds_staged && ok && n_iter > 0) {
                    ok = mbar_wait(&bars[Cfg::kBiasEmpty], (uint32_t)(done - 1) & 1u, abort_flag);
                    if (ok) store_ds(n_iter - 1);
                }
            }
            for (int spin = 0; !ok && spin < 4096 && done > 0 && !mbar_try_wait(&bars[Cfg::kBiasFull], (uint32_t)(done - 1) & 1u); ++spin) {}
        }
        __syncwarp();
      }
    } else {
        // ---------------------------------------------------------------- P / dS and epilogue
        if constexpr (kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsElementwiseMoved));
        constexpr int NLD = CPT / 32;                          // 32-column TMEM loads per thread and phase
        const int wg = warp >> 2;                              // which CPT-column slice
        const int r = (warp & 3) * 32 + lane;                  // TMEM lane = row of T1/T2
        const int cb = wg * CPT;
        const int tid = wg * 128 + r;                          // 0 .. 128*NWG-1
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        constexpr bool drop = DROP != 0;
        // bf16: a stationary tile to fp16 in place (K_j and V_j, or Q_i; dO_i is only ever multiplied with the bf16 V_j
        // tiles and stays as it is), by all elementwise warps: a block's X while the one before it still waits for its
        // accumulators, its Y behind that one's epilogue.  By the two spare warps it took 4000 cycles a tile.
        auto convert_xy = [&](int y, uint32_t parity) {
            bool good = mbar_wait(&bars[Cfg::kXFull + y], parity, abort_flag);
            good = __all_sync(0xffffffffu, good);
            if (!good) return false;
            convert_tile_bf16_to_f16<false>(sX + y * TILE, TILE, tid, 128 * NWG, 1.f);
            fence_proxy_async_smem();
            mbar_arrive_warp(&bars[Cfg::kXConv + y]);
            return true;
        };
        bool ok = true;
        int g = 0;                           // steps so far
        uint32_t count = 0u;                 // blocks (bits 0-1), blocks with steps (bit 2): as much as the barriers' phases need
        ok = __all_sync(0xffffffffu, item_there(0));
        if (XY_CONV && ok && sched[0].n_iter > 0) ok = convert_xy(0, 0u);
        auto scales = [&](const volatile BwdItem* m) {
            const float range[2] = {m->range[0], m->range[1]};
            return make_scales(range, D, a.inv_keep, a.scale, kForm);
        };
        while (ok) {
        [[maybe_unused]] BwdScales sc_row;       // ROW_MAX: the row's own
        {
        const volatile BwdItem* m = sched + (count & 1u);
        const int tile = m->tile, head_x = m->head_x, b = m->b, nk = m->nk, it0 = m->it0, n_per_head = m->n_per_head, n_iter = m->n_iter;
        [[maybe_unused]] const int sum_steps = DS ? n_per_head : 0;
        [[maybe_unused]] const int rot = FUSED ? m->rot : 0;
        if (n_iter < 0) break;
        if (XY_CONV && KS && n_iter > 0) {
            ok = convert_xy(1, (count >> 2) & 1u);
            if (!ok) break;
        }
        const int row_g = tile * kTile + r;                    // MODE 0: key index; MODE 1: query index
        BwdScales sc = scales(m);
        float my_nlse2 = 0.f, my_ndelta = 0.f;      // -lse*log2(e) and -delta of my query row (MODE 1)
        if (MODE == 1 && n_iter > 0) {
            ok = mbar_wait(&bars[Cfg::kRowFull], (count >> 2) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            my_nlse2 = sVec[r];
            my_ndelta = sVec[128 + r];
            const float e = ROWFORM ? sVec[256 + r] : 0.f;
            if (!DS) mbar_arrive_read_done(&bars[Cfg::kRowEmpty]);       // (else its room holds sums first)
            if (ROWFORM) {
                // the vectors are staged for the key-stationary kernels: take the row exponent out again
                const int e_i = (int)e;
                my_nlse2 -= (float)e_i;            // -inf in the padding stays -inf
                my_ndelta *= pow2i(e_i);
            }
            // pairs: P = 2^((S scale + bias - lse) log2 e) 2^kPShift with the terms in the forward's order, so that a mask
            // of the type's lowest value or of -1e9 leaves in both what its rounding leaves (the difference is small
            // wherever P is not), and the shift (fp16 only) exact behind it: d(loss)/d(scores) is an fp32 result.
        }
        if constexpr (ROW_MAX) {
            // fp16 pairs: dS of my row scaled by a power of two of its own, from its own max |dO|, so that rows far
            // below the column's largest keep their bits (dQ and d(loss)/d(scores) of a row need no common scale; the
            // other kernel sums over rows and has to have one)
            if (n_iter > 0) ok = mbar_wait(&bars[Cfg::kYFull], (count >> 2) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (n_iter > 0 && ok) {
                uint32_t top = 0u;
#pragma unroll
                for (int c = 0; c < Cfg::kNBox * 8; ++c) {
                    const uint32_t mp = finite_piece<__half>(absmax16_acc(
                        0u, *reinterpret_cast<const uint4*>(sY + (c >> 3) * kBoxBytes + r * 128 + (((c ^ r) & 7) << 4))));
                    asm("max.u16x2 %0, %0, %1;" : "+r"(top) : "r"(mp));
                }
                const float rng[2] = {__half2float(__ushort_as_half((unsigned short)max(top & 0xFFFFu, top >> 16))), m->range[1]};
                sc = make_scales(rng, D, a.inv_keep, a.scale, kDoAsIs);
                mbar_arrive_read_done(&bars[Cfg::kYEmpty]);
            }
        }
        // dS' = P' o (dP * tt_mul o Z + (-delta) * nd_mul): see "number formats" above
        const float tt_mul = DS ? sc.tt_mul * a.dp_gain : sc.tt_mul;
        const uint64_t ttm2 = f2_pack(tt_mul, tt_mul), ndm2 = f2_pack(sc.nd_mul, sc.nd_mul);
        const float zk = a.inv_keep * tt_mul;
        const uint64_t ladd2 = f2_pack(sc.l_add, sc.l_add);
        my_ndelta *= sc.nd_mul;
        // PREC = 1, query-stationary: my row of d loss / d scores, and what undoes dS' = dS * 2^g
        [[maybe_unused]] float* ds_row = DS
            ? a.d_scores + (((int64_t)b * a.H + head_x) * a.Nq + row_g) * (int64_t)a.Nk : nullptr;
        [[maybe_unused]] const float ds_mul = sc.ds_mul;
        // fused kernel: add the dQ tile of step `jt` (queries on the TMEM lanes, my D / NWG columns)
        // to the fp32 sums in global memory; the order of additions across CTAs is not fixed
        auto drain_dq = [&](int jt, int q_tile, int head_q) -> bool {
            constexpr int DQC = D / NWG;
            bool good = mbar_wait(&bars[Cfg::kDqFull], (uint32_t)jt & 1u, abort_flag);
            good = __all_sync(0xffffffffu, good);
            if (!good) return false;
            tc_fence_after_sync();
            uint32_t acc[DQC];
            if constexpr (DQC == 32) tmem_ld_32x32(tDq + lane_off + (uint32_t)(wg * DQC), acc);
            else                     tmem_ld_32x16(tDq + lane_off + (uint32_t)(wg * DQC), acc);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[Cfg::kDqRead]);
            float* dst = a.dq_acc + (((int64_t)b * a.H + head_q) * (a.nq_pad / kTile) + q_tile) * (int64_t)(kTile * D) +
                         ((int64_t)(wg * (DQC / 4)) * kTile + r) * 4;
#pragma unroll
            for (int v = 0; v < DQC / 4; ++v)
                red_add_v4_f32(dst + (int64_t)v * kTile * 4, __uint_as_float(acc[4 * v]), __uint_as_float(acc[4 * v + 1]),
                               __uint_as_float(acc[4 * v + 2]), __uint_as_float(acc[4 * v + 3]));
            return true;
        };

        // Pairs with d(loss)/d(scores) wanted (MODE 1).  That output is fp32, but delta comes from an O rounded to 16 bits
        // (or 16 + 16) that was summed with P as a pair, and P from an lse rounded once: together more than the CUDA
        // cores' error.  So a first walk over the keys sums P and P o dP Z of every row in fp32; their quotient is
        // delta, and the sum of P, one but for rounding, divides P (distance from float64 at B2 N440 H4 D64 bf16, CUDA cores
        // 3.5e-7: 5.6e-7 -> 2.4e-7; N385 causal 1.05e-6: 1.23e-6 -> 1.8e-7).
        [[maybe_unused]] uint64_t sum_p2 = 0ull, sum_pd2 = 0ull;           // {0.f, 0.f}
        [[maybe_unused]] float p_mul = P_BF16 ? 1.f : 16384.f;             // 2^kPShift where P carries it
        int qi = 0, hg = 0;                 // step within the query head, query heads done (key-stationary)
        int prev_tile = 0, prev_head = 0;   // query tile and head of the previous step
        for (const int g0 = g, g_end = g + n_iter; g < g_end && ok; ++g) {
            const int it = g - g0;          // (query-stationary)
            const int strm_tile = (KS) ? q_tile_of(it0, n_per_head, rot, qi) : k_tile_of(n_per_head, it);     // query tile (0) / key tile (1)
            const int col_g0 = strm_tile * kTile + cb;                          // global index of my first column
            const int head_q = (KS) ? head_x * a.group + hg : head_x;
            const uint32_t bh = dropout_column(a.rng, b, head_q);
            [[maybe_unused]] const float* bias_h = PREC ? a.bias + b * a.bias_sb + head_q * a.bias_sh : nullptr;
            // key-stationary: -lse*log2(e) and -delta of this step's 128 queries (slot g & 1)
            const float* lse_s = sVec + (g & 1) * 256;
            const float* del_s = lse_s + 128;

            // ---- dropout keep bits of my CPT columns (bit c of kb[c / 32])
            uint32_t kb[2] = {0xFFFFFFFFu, 0xFFFFFFFFu};
            if (drop) {
                kb[0] = 0u; kb[1] = 0u;
                if constexpr (DROP == 2) {
                    static_assert(CPT % 32 == 0, "a thread's columns are whole words of the bit buffer");
                    if (MODE == 1) {
                        // my query row's bits for this key tile: the words of my CPT columns
                        const uint32_t* w = reinterpret_cast<const uint32_t*>(
                            a.bits_q + ((int64_t)(b * a.H + head_q) * (a.nk_pad / kTile) + strm_tile) * a.nq_pad + row_g);
#pragma unroll
                        for (int g = 0; g < CPT / 32; ++g) kb[g] = w[cb / 32 + g];
                    } else if (FUSED) {
                        // my key row's bits for this query tile, 32 queries a word
                        const uint32_t* w = a.bits_k + (((int64_t)(b * a.H + head_q) * (a.nq_pad / kTile) + strm_tile) * 4 +
                                                        cb / 32) * (int64_t)a.nk_pad + row_g;
#pragma unroll
                        for (int g = 0; g < CPT / 32; ++g) kb[g] = w[(int64_t)g * a.nk_pad];
                    }
                } else if (MODE == 1) {
#pragma unroll
                    for (int g = 0; g < CPT / 16; ++g) {
                        const uint32_t w = dropout_keep_bits(a.key, bh, (uint32_t)row_g, (uint32_t)((col_g0 >> 4) + g),
                                                             a.drop_thr);
                        kb[g >> 1] |= w << (16 * (g & 1));
                    }
                } else {
                    // keys are rows here: build the tile's masks cooperatively, query-major, then read
                    // one bit per (query column, my key row)
                    constexpr int PER = 8 / NWG;               // 16-key blocks each thread generates
                    uint16_t* mbuf = sMask + (g & 1) * (128 * 8);
                    const int ql = tid & 127, jb0 = (tid >> 7) * PER;
#pragma unroll
                    for (int q = 0; q < PER; ++q)
                        mbuf[ql * 8 + jb0 + q] = (uint16_t)dropout_keep_bits(
                            a.key, bh, (uint32_t)(strm_tile * kTile + ql), (uint32_t)(tile * 8 + jb0 + q), a.drop_thr);
                    mbar_arrive_warp(&bars[Cfg::kMask]);
                    ok = mbar_wait(&bars[Cfg::kMask], (uint32_t)g & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (FUSED) {      // (the fragment-layout phases read their keep bits from mbuf themselves)
                        const int jw = r >> 4, jbit = r & 15;
#pragma unroll
                        for (int c = 0; c < CPT; ++c)
                            kb[c >> 5] |= (((uint32_t)mbuf[(cb + c) * 8 + jw] >> jbit) & 1u) << (c & 31);
                    }
                }
            }

            if constexpr (MODE == 0) {
            // ---- dK/dV kernel, fragment layout: a thread holds 4 rows x 8 columns of its warp's
            // 32 x 32 block (rows lane/4 + {0, 8, 16, 24}, columns 8j + 2(lane%4) + {0, 1}, j = 0..3) instead
            // of 1 row x 32 columns, so it needs the -lse / -delta values of 8 query columns, four 8-byte
            // loads that one wavefront serves, instead of 32 values through eight broadcast 16-byte loads.
            const int lq = lane & 3, lr = lane >> 2;
            const int rbase = (warp & 3) * 32 + lr;                 // my first row inside the tile
            // DROP = 2: one word of keep bits per key row of mine, asked for before the wait for S^T
            uint32_t kwr[2][2] = {{0u, 0u}, {0u, 0u}};
            if constexpr (DROP == 2) {
                const uint32_t* w = a.bits_k + (((int64_t)(b * a.H + head_q) * (a.nq_pad / kTile) + strm_tile) * 4 +
                                                cb / 32) * (int64_t)a.nk_pad + tile * kTile + rbase;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < 2; ++k) kwr[h][k] = w[16 * h + 8 * k];
            }
            ok = mbar_wait(&bars[Cfg::kT1Full], (uint32_t)g & 1u, abort_flag);
            if (ok) ok = mbar_wait(&bars[Cfg::kVFull + (g & 1)], (uint32_t)(g >> 1) & 1u, abort_flag);
            if (PREC == 2 && ok) ok = mbar_wait(&bars[Cfg::kBiasFull], (uint32_t)g & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t t_lo = lane_off + cb, t_hi = lane_off + (16u << 16) + cb;
            // element (h, j, k, e): row rbase + 16h + 8k, column 8j + 2lq + e, register [h][4j + 2k + e]
            uint32_t pf[2][16];
            tmem_ld_16x256b_x4(tT1 + t_lo, pf[0]);
            tmem_ld_16x256b_x4(tT1 + t_hi, pf[1]);
            tmem_wait_ld();
            uint32_t kbits = 0xFFFFFFFFu;                           // keep bit of element (h, j, k, e): bit 16h + 4j + 2k + e
            if constexpr (DROP == 2) {
                // shifted so that bit 8j + e is my column 8j + 2lq + e
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < 2; ++k) kwr[h][k] >>= ((cb & 31) + 2 * lq);
            } else if (drop) {
                const uint16_t* mbuf = sMask + (g & 1) * (128 * 8);
                kbits = 0u;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int row = rbase + 16 * h + 8 * k, col = cb + 8 * j + 2 * lq + e;
                                kbits |= (((uint32_t)mbuf[col * 8 + (row >> 4)] >> (row & 15)) & 1u) << (16 * h + 4 * j + 2 * k + e);
                            }
            }
            const float sc1 = PREC ? a.score_scale : a.scale_log2;
            const uint64_t sc2 = f2_pack(sc1, sc1);
            // key row > query column + shift is hidden: only tiles the mask's edge crosses need the test
            const bool diag = a.causal && strm_tile * kTile + a.shift < tile * kTile + kTile - 1;
            const bool tail = tile * kTile + kTile > nk;            // the tile holds padding keys
            // query columns below `lim` do not see a key row: all of them for a
            // padding key, those with column + shift < row under the mask's edge
            auto hidden_below = [&](int h, int k) {
                const int row_k = tile * kTile + rbase + 16 * h + 8 * k;
                return (tail && row_k >= nk) ? 0x7fffffff : (diag ? row_k - a.shift : -0x7fffffff);
            };
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t pk[2][4], pl[2][4];                        // [h][2j' + k], j' = j - 2hf; pairs: the low parts
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    const int j = 2 * hf + jj;
                    if (!drop && hf == 1 && jj == 0) {
                        // hand the first half over before the second is computed, so that its MMAs are done
                        // when the second half arrives (dK/dV 0.971 -> 0.933 ms at B4 N4096 H32 D128: the chain
                        // MMA -> threads -> MMA feels every cycle).  With dropout the threads are the slower
                        // side and the wait for the stores just issued costs more than it gains (1.24 against
                        // 1.22 ms at B32 N2048 H16 D64): there the hand-off stays behind the second half's math.
                        tmem_wait_st();
                        tc_fence_before_sync();
                        mbar_arrive_warp(&bars[Cfg::kPHalf]);
                    }
                    uint64_t L = *reinterpret_cast<const uint64_t*>(lse_s + cb + 8 * j + 2 * lq);
                    if (ROWFORM) L = f2_add(L, ladd2);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int i0 = 4 * j + 2 * k;
                            float x0, x1;
                            uint64_t add = L;                  // pairs with a bias: the bias first, in natural units, then -lse
                            float b0 = 0.f, b1 = 0.f;
                            if constexpr (PREC == 2) {
                                // bias[query][key] from the tile: eight keys (two 16-byte pieces) of four queries a load,
                                // which the swizzle spreads over all banks
                                const int kk = lr + 16 * h + 8 * k;
                                const uint8_t* bp = sBias + (warp & 3) * kBoxBytes + (cb + 8 * j + 2 * lq) * 128 + (kk & 3) * 4;
                                b0 = *reinterpret_cast<const float*>(bp + (((kk >> 2) ^ (2 * lq)) << 4));
                                b1 = *reinterpret_cast<const float*>(bp + 128 + (((kk >> 2) ^ (2 * lq + 1)) << 4));
                            } else if (PREC && a.bias) {
                                // bias[query][key]: eight lanes read eight neighbouring keys of one query
                                const int key = tile * kTile + rbase + 16 * h + 8 * k, qr = col_g0 + 8 * j + 2 * lq;
                                const float* bp = bias_h + (int64_t)qr * a.bias_sn + key;
                                if (key < a.Nk && qr < a.Nq) b0 = bp[0];
                                if (key < a.Nk && qr + 1 < a.Nq) b1 = bp[a.bias_sn];
                            }
                            if (PREC == 2 || (PREC == 1 && a.bias)) add = f2_pack(b0, b1);
                            uint64_t x = f2_fma(f2_pack(__uint_as_float(pf[h][i0]), __uint_as_float(pf[h][i0 + 1])), sc2, add);
                            if (PREC == 2 || (PREC == 1 && a.bias)) x = f2_add(x, L);
                            if (P_BF16)    x = f2_mul(x, f2_pack(kLog2e, kLog2e));
                            else if (PREC) x = f2_fma(x, f2_pack(kLog2e, kLog2e), f2_pack(kPShift, kPShift));
                            f2_unpack(x, x0, x1);
                            pf[h][i0] = __float_as_uint(ex2(x0));
                            pf[h][i0 + 1] = __float_as_uint(ex2(x1));
                        }
                }
                if (PREC == 2 && hf == 1) mbar_arrive_read_done(&bars[Cfg::kBiasEmpty]);
                if (diag || tail) {
                    // one branch for the whole half: the diagonal tile and a tile with padding keys are rare
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const int j = 2 * hf + jj, i0 = 4 * j + 2 * k;
                                const int col = col_g0 + 8 * j + 2 * lq, lim = hidden_below(h, k);
                                if (col < lim) pf[h][i0] = 0u;
                                if (col + 1 < lim) pf[h][i0 + 1] = 0u;
                            }
                }
#pragma unroll
                for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int i0 = 4 * (2 * hf + jj) + 2 * k;
                            float z0 = __uint_as_float(pf[h][i0]), z1 = __uint_as_float(pf[h][i0 + 1]);
                            if (drop) {
                                const uint32_t kw = DROP == 2 ? kwr[h][k] >> (8 * (i0 >> 2)) : kbits >> (16 * h + i0);
                                if (!(kw & 1u)) z0 = 0.f;
                                if (!(kw & 2u)) z1 = 0.f;
                            }
                            if (PREC) pack2_pair<P_BF16>(z0, z1, pk[h][2 * jj + k], pl[h][2 * jj + k]);
                            else      pk[h][2 * jj + k] = pack2<false>(z0, z1);
                        }
                if (drop && hf == 1) {
                    tmem_wait_st();
                    tc_fence_before_sync();
                    mbar_arrive_warp(&bars[Cfg::kPHalf]);
                }
                tmem_st_16x128b_x2(tT1 + t_lo + hf * 8, pk[0]);
                tmem_st_16x128b_x2(tT1 + t_hi + hf * 8, pk[1]);
                if (PREC) {
                    tmem_st_16x128b_x2(tT1 + t_lo + 16 + hf * 8, pl[0]);
                    tmem_st_16x128b_x2(tT1 + t_hi + 16 + hf * 8, pl[1]);
                }
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[Cfg::kPReady]);

            ok = mbar_wait(&bars[Cfg::kT2Full], (uint32_t)g & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            {
                uint32_t df[2][16];
                tmem_ld_16x256b_x4(tT2 + t_lo, df[0]);
                tmem_ld_16x256b_x4(tT2 + t_hi, df[1]);
                tmem_wait_ld();
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t pk[2][4], pl[2][4];
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        const int j = 2 * hf + jj;
                        if (!drop && hf == 1 && jj == 0) {
                            tmem_wait_st();                        // the first half, as for P above
                            tc_fence_before_sync();
                            mbar_arrive_warp(&bars[Cfg::kDsHalf]);
                        }
                        const uint64_t nd = f2_mul(*reinterpret_cast<const uint64_t*>(del_s + cb + 8 * j + 2 * lq), ndm2);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const int i0 = 4 * j + 2 * k;
                                const uint64_t dp = f2_pack(__uint_as_float(df[h][i0]), __uint_as_float(df[h][i0 + 1]));
                                uint64_t tt;
                                if (drop) {
                                    const uint32_t kw = DROP == 2 ? kwr[h][k] >> (8 * j) : kbits >> (16 * h + i0);
                                    tt = f2_fma(dp, f2_pack((kw & 1u) ? zk : 0.f, (kw & 2u) ? zk : 0.f), nd);
                                } else {
                                    tt = f2_fma(dp, ttm2, nd);
                                }
                                float d0, d1;
                                f2_unpack(f2_mul(f2_pack(__uint_as_float(pf[h][i0]), __uint_as_float(pf[h][i0 + 1])), tt), d0, d1);
                                // as in the other kernel: none, not 0 times what delta is (only a bias makes rows without a result)
                                if ((PREC == 2 || (PREC == 1 && a.bias)) && (diag || tail)) {
                                    const int col = col_g0 + 8 * j + 2 * lq, lim = hidden_below(h, k);
                                    if (col < lim) d0 = 0.f;
                                    if (col + 1 < lim) d1 = 0.f;
                                }
                                if (PREC) pack2_pair<P_BF16>(d0, d1, pk[h][2 * jj + k], pl[h][2 * jj + k]);
                                else      pk[h][2 * jj + k] = pack2<false>(d0, d1);
                            }
                    }
                    if (drop && hf == 1) {
                        tmem_wait_st();
                        tc_fence_before_sync();
                        mbar_arrive_warp(&bars[Cfg::kDsHalf]);
                    }
                    tmem_st_16x128b_x2(tT2 + t_lo + hf * 8, pk[0]);
                    tmem_st_16x128b_x2(tT2 + t_hi + hf * 8, pk[1]);
                    if (PREC) {
                        tmem_st_16x128b_x2(tT2 + t_lo + 16 + hf * 8, pl[0]);
                        tmem_st_16x128b_x2(tT2 + t_hi + 16 + hf * 8, pl[1]);
                    }
                }
                tmem_wait_st();
            }
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[Cfg::kDsReady]);
            } else {
            // ---- one row and 32 columns per thread: the query-stationary kernel (lse and delta are
            // per-thread scalars there), and the one-kernel backward, whose dS^T tile for the dQ MMA is
            // written with 16-byte stores from this layout (with the fragment layout above it measured
            // 5-10 % slower)
            // ---- phase A: P from T1
            ok = mbar_wait(&bars[Cfg::kT1Full], (uint32_t)g & 1u, abort_flag);
            if (KS && ok) ok = mbar_wait(&bars[Cfg::kVFull + (g & 1)], (uint32_t)(g >> 1) & 1u, abort_flag);
            if (PREC == 2 && ok) ok = mbar_wait(&bars[Cfg::kBiasFull], (uint32_t)g & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            uint32_t pr[NLD][32];      // P of my columns (fp32 bits), kept for phase B
#define PF(c) __uint_as_float(pr[(c) >> 5][(c) & 31])
#define PSET(c, x) pr[(c) >> 5][(c) & 31] = __float_as_uint(x)
#pragma unroll
            for (int q = 0; q < NLD; ++q) tmem_ld_32x32(tT1 + lane_off + cb + q * 32, pr[q]);
            tmem_wait_ld();
            if (!KS) {
                // query-stationary: P stays in registers, so S's columns are free for S(it+1) from here on
                tc_fence_before_sync();
                mbar_arrive_warp(&bars[Cfg::kPReady]);
            }
            const uint64_t sc2 = f2_pack(a.scale_log2, a.scale_log2);
            [[maybe_unused]] const bool summing = DS && it < sum_steps;
            [[maybe_unused]] int seen = CPT;           // pairs, query-stationary: my first columns that my row sees
            if (KS) {
                // P = 2^(S*c - lse): the staged vector holds -lse*log2(e), two columns per 64-bit word.
                // Two halves of CPT / 2 columns: the first is packed, stored to TMEM and handed to the
                // MMA warp (dV can start on it) while the second is computed.
                static_assert(CPT == 32, "the half hand-off is written for 32 columns per thread");
                const ulonglong2* l2 = reinterpret_cast<const ulonglong2*>(lse_s + cb);
                const bool diag = a.causal && strm_tile * kTile + a.shift < tile * kTile + kTile - 1;
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    if (hf == 1) {
                        // hand the first half over before the second is computed: its MMAs are then done
                        // when the second half arrives (the chain MMA -> threads -> MMA feels every cycle)
                        tmem_wait_st();
                        tc_fence_before_sync();
                        mbar_arrive_warp(&bars[Cfg::kPHalf]);
                    }
#pragma unroll
                    for (int c4 = hf * (CPT / 8); c4 < (hf + 1) * (CPT / 8); ++c4) {
                        ulonglong2 L = l2[c4];
                        if (ROWFORM) { L.x = f2_add(L.x, ladd2); L.y = f2_add(L.y, ladd2); }
                        float x0, x1, x2, x3;
                        f2_unpack(f2_fma(f2_pack(PF(c4 * 4 + 0), PF(c4 * 4 + 1)), sc2, L.x), x0, x1);
                        f2_unpack(f2_fma(f2_pack(PF(c4 * 4 + 2), PF(c4 * 4 + 3)), sc2, L.y), x2, x3);
                        PSET(c4 * 4 + 0, ex2(x0));
                        PSET(c4 * 4 + 1, ex2(x1));
                        PSET(c4 * 4 + 2, ex2(x2));
                        PSET(c4 * 4 + 3, ex2(x3));
                    }
                    if (diag) {
                        const int hidden = row_g - col_g0 - a.shift;   // my first `hidden` columns: query + shift < key
#pragma unroll
                        for (int c = hf * (CPT / 2); c < (hf + 1) * (CPT / 2); ++c)
                            if (c < hidden) PSET(c, 0.f);
                    }
                    if (row_g >= nk) {                    // a padding key inside a live tile (or beyond Nk)
#pragma unroll
                        for (int c = hf * (CPT / 2); c < (hf + 1) * (CPT / 2); ++c) PSET(c, 0.f);
                    }
                    uint32_t pk[CPT / 4];
#pragma unroll
                    for (int e = 0; e < CPT / 4; ++e) {
                        const int c = hf * (CPT / 2) + 2 * e;
                        float x0 = PF(c), x1 = PF(c + 1);
                        if (drop) {
                            if (!((kb[c >> 5] >> (c & 31)) & 1u)) x0 = 0.f;
                            if (!((kb[(c + 1) >> 5] >> ((c + 1) & 31)) & 1u)) x1 = 0.f;
                        }
                        pk[e] = pack2<false>(x0, x1);
                    }
                    tmem_st_32x8(tT1 + lane_off + cb + hf * (CPT / 4), pk);
                }
                tmem_wait_st();
            } else {
                const uint64_t neg2 = f2_pack(my_nlse2, my_nlse2);
                [[maybe_unused]] const uint64_t scn2 = f2_pack(a.score_scale, a.score_scale), log2e2 = f2_pack(kLog2e, kLog2e), up2 = f2_pack(p_mul, p_mul);
                [[maybe_unused]] float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int c = 0; c < CPT; c += 2) {
                    float x0, x1;
                    if constexpr (PREC != 0) {
                        const uint64_t s2 = f2_pack(PF(c), PF(c + 1));
                        uint64_t x;
                        if (PREC == 2 || a.bias) {
                            float b0 = 0.f, b1 = 0.f;
                            if constexpr (PREC == 2) {
                                // my row's 32 keys are the wg-th box, its 16-byte pieces swizzled by the row
                                if ((c & 3) == 0) bv = *reinterpret_cast<const float4*>(sBias + wg * kBoxBytes + r * 128 + (((c >> 2) ^ (r & 7)) << 4));
                                b0 = (c & 2) ? bv.z : bv.x;
                                b1 = (c & 2) ? bv.w : bv.y;
                            } else {
                                const float* bp = bias_h + (int64_t)(row_g < a.Nq ? row_g : a.Nq - 1) * a.bias_sn + col_g0 + c;
                                if (a.bias_vec && col_g0 + (c & ~3) + 4 <= a.Nk) {
                                    if ((c & 3) == 0) bv = *reinterpret_cast<const float4*>(bp);
                                    b0 = (c & 2) ? bv.z : bv.x;
                                    b1 = (c & 2) ? bv.w : bv.y;
                                } else {
                                    if (col_g0 + c < a.Nk) b0 = bp[0];
                                    if (col_g0 + c + 1 < a.Nk) b1 = bp[1];
                                }
                            }
                            x = f2_add(f2_fma(s2, scn2, f2_pack(b0, b1)), neg2);
                        } else {
                            x = f2_fma(s2, scn2, neg2);
                        }
                        f2_unpack(f2_mul(x, log2e2), x0, x1);
                        x0 = ex2(x0);
                        x1 = ex2(x1);
                        if (DS || !P_BF16) f2_unpack(f2_mul(f2_pack(x0, x1), up2), x0, x1);
                        PSET(c, x0);
                        PSET(c + 1, x1);
                        continue;
                    }
                    f2_unpack(f2_fma(f2_pack(PF(c), PF(c + 1)), sc2, neg2), x0, x1);
                    // a quarter of the exponentials as a polynomial on the FMA pipes (this kernel keeps the
                    // special-function unit busiest; measured 0.7 % over the backward, half: 0.2 %)
                    if (((c >> 1) & 3) == 0) {
                        float p0, p1;
                        ex2_poly2(x0, x1, p0, p1);
                        PSET(c, p0);
                        PSET(c + 1, p1);
                    } else {
                        PSET(c, ex2(x0));
                        PSET(c + 1, ex2(x1));
                    }
                }
                if (PREC == 2 && (!DS || !a.ds_staged || summing)) mbar_arrive_read_done(&bars[Cfg::kBiasEmpty]);
                const bool diag = a.causal && strm_tile * kTile + kTile - 1 > tile * kTile + a.shift;
                if (diag || strm_tile * kTile + kTile > nk) {
                    // my row sees my first `seen` columns: keys below the count, at most row + shift
                    seen = nk - col_g0;
                    if (diag && row_g + a.shift + 1 - col_g0 < seen) seen = row_g + a.shift + 1 - col_g0;
#pragma unroll
                    for (int c = 0; c < CPT; ++c)
                        if (c >= seen) PSET(c, 0.f);
                }
            }
            if (KS) {
                tc_fence_before_sync();
                mbar_arrive_warp(&bars[Cfg::kPReady]);
            }

            if (FUSED && qi + hg > 0) {
                // dQ of the previous step: its MMAs ran while phase A above did
                ok = drain_dq(g - 1, prev_tile, prev_head);
                if (!ok) break;
            }

            // ---- phase B: dS from T2
            // query-stationary: dP / dS alternate between two buffers, each with its own barriers
            const bool odd_buf = !KS && (g & 1);
            const uint32_t tD = odd_buf ? tAcc2 : tT2;
            const int b_half = odd_buf ? Cfg::kPHalf : Cfg::kDsHalf, b_ready = odd_buf ? Cfg::kDqRead : Cfg::kDsReady;
            ok = KS ? mbar_wait(&bars[Cfg::kT2Full], (uint32_t)g & 1u, abort_flag)
                    : mbar_wait(&bars[odd_buf ? Cfg::kT1Full + 1 : Cfg::kT2Full], (uint32_t)(g >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            {
                uint32_t dr[NLD][32];
#pragma unroll
                for (int q = 0; q < NLD; ++q) tmem_ld_32x32(tD + lane_off + cb + q * 32, dr[q]);
                tmem_wait_ld();
                // dS = P o (dP o Z - delta); the staged vector holds -delta.  Two halves, as in phase A:
                // the first is stored and handed over while the second is computed.
                const ulonglong2* d2 = reinterpret_cast<const ulonglong2*>(del_s + cb);
                const uint64_t my_nd2 = f2_pack(my_ndelta, my_ndelta);
                if (summing) {
                    tc_fence_before_sync();
                    mbar_arrive_warp(&bars[b_half]);
                    uint64_t sp = 0ull, spd = 0ull;
#pragma unroll
                    for (int c = 0; c < CPT; c += 2) {
                        const uint64_t p2 = f2_pack(PF(c), PF(c + 1));
                        uint64_t z2 = ttm2;
                        if (drop) z2 = f2_pack(((kb[0] >> c) & 1u) ? zk : 0.f, ((kb[0] >> c) & 2u) ? zk : 0.f);
                        sp = f2_add(sp, p2);
                        uint64_t t2 = f2_mul(p2, f2_mul(f2_pack(__uint_as_float(dr[0][c]), __uint_as_float(dr[0][c + 1])), z2));
                        if (seen < CPT) {              // hidden: no part of the sum, also where dP is no number
                            float t0, t1;
                            f2_unpack(t2, t0, t1);
                            t2 = f2_pack(c < seen ? t0 : 0.f, c + 1 < seen ? t1 : 0.f);
                        }
                        spd = f2_add(spd, t2);
                    }
                    sum_p2 = f2_add(sum_p2, sp);
                    sum_pd2 = f2_add(sum_pd2, spd);
                } else {
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t pk[CPT / 4], pl[CPT / 4];
                        if (hf == 1) {
                            tmem_wait_st();                            // the first half, stored just now
                            tc_fence_before_sync();
                            mbar_arrive_warp(&bars[b_half]);
                        }
#pragma unroll
                        for (int c4 = hf * (CPT / 8); c4 < (hf + 1) * (CPT / 8); ++c4) {
                            ulonglong2 nd;
                            if (KS) { nd = d2[c4]; nd.x = f2_mul(nd.x, ndm2); nd.y = f2_mul(nd.y, ndm2); }
                            else { nd.x = my_nd2; nd.y = my_nd2; }
                            const int c = c4 * 4;
                            uint64_t dpa = f2_pack(__uint_as_float(dr[c >> 5][c & 31]), __uint_as_float(dr[c >> 5][(c + 1) & 31]));
                            uint64_t dpb = f2_pack(__uint_as_float(dr[c >> 5][(c + 2) & 31]), __uint_as_float(dr[c >> 5][(c + 3) & 31]));
                            uint64_t ta, tb;
                            if (drop) {
                                // dropped entries: dS = P o (-delta), selected after the FMA
                                const uint32_t kw = kb[c >> 5] >> (c & 31);
                                const uint64_t zk2 = f2_pack(zk, zk);
                                float t0, t1, t2, t3, n0, n1, n2, n3;
                                f2_unpack(f2_fma(dpa, zk2, nd.x), t0, t1);
                                f2_unpack(f2_fma(dpb, zk2, nd.y), t2, t3);
                                f2_unpack(nd.x, n0, n1);
                                f2_unpack(nd.y, n2, n3);
                                ta = f2_pack((kw & 1u) ? t0 : n0, (kw & 2u) ? t1 : n1);
                                tb = f2_pack((kw & 4u) ? t2 : n2, (kw & 8u) ? t3 : n3);
                            } else {
                                ta = f2_fma(dpa, ttm2, nd.x);
                                tb = f2_fma(dpb, ttm2, nd.y);
                            }
                            float d0, d1, d2v, d3;
                            f2_unpack(f2_mul(f2_pack(PF(c), PF(c + 1)), ta), d0, d1);
                            f2_unpack(f2_mul(f2_pack(PF(c + 2), PF(c + 3)), tb), d2v, d3);
                            if constexpr (PREC != 0) {
                                // a hidden score has no gradient, also where delta or dP is no number (0 times that is none)
                                if (DS && seen < CPT) {
                                    if (c >= seen) d0 = 0.f;
                                    if (c + 1 >= seen) d1 = 0.f;
                                    if (c + 2 >= seen) d2v = 0.f;
                                    if (c + 3 >= seen) d3 = 0.f;
                                }
                                const int e = (c4 - hf * (CPT / 8)) * 2;
                                pack2_pair<P_BF16>(d0, d1, pk[e], pl[e]);
                                pack2_pair<P_BF16>(d2v, d3, pk[e + 1], pl[e + 1]);
                                if (DS && PREC == 2 && a.ds_staged) {
                                    // ... by way of the bias tile's place (only I read these 16 bytes) and a TMA store: a
                                    // thread's own stores would go to 32 rows a warp
                                    *reinterpret_cast<float4*>(sBias + wg * kBoxBytes + r * 128 + (((c >> 2) ^ (r & 7)) << 4)) =
                                        make_float4(d0 * ds_mul, d1 * ds_mul, d2v * ds_mul, d3 * ds_mul);
                                } else if (DS && row_g < a.Nq) {
                                    // d loss / d scores, the power of two of dS' taken out (exact)
                                    float* dst = ds_row + col_g0 + c;
                                    if (a.ds_vec) {
                                        if (col_g0 + c < a.Nk)
                                            *reinterpret_cast<float4*>(dst) = make_float4(d0 * ds_mul, d1 * ds_mul, d2v * ds_mul, d3 * ds_mul);
                                    } else {
                                        if (col_g0 + c < a.Nk) dst[0] = d0 * ds_mul;
                                        if (col_g0 + c + 1 < a.Nk) dst[1] = d1 * ds_mul;
                                        if (col_g0 + c + 2 < a.Nk) dst[2] = d2v * ds_mul;
                                        if (col_g0 + c + 3 < a.Nk) dst[3] = d3 * ds_mul;
                                    }
                                }
                            } else {
                                pk[(c4 - hf * (CPT / 8)) * 2 + 0] = pack2<false>(d0, d1);
                                pk[(c4 - hf * (CPT / 8)) * 2 + 1] = pack2<false>(d2v, d3);
                            }
                        }
                        tmem_st_32x8(tD + lane_off + cb + hf * (CPT / 4), pk);
                        if (PREC) tmem_st_32x8(tD + lane_off + cb + CPT / 2 + hf * (CPT / 4), pl);
                        if (FUSED) {
                            // the same dS^T values as a shared-memory tile [key row][query], 64-query boxes with
                            // the 128-byte swizzle: the A operand (MN-major) of the dQ MMA.  The previous
                            // step's dQ MMA has finished reading it: its completion was awaited in drain_dq.
#pragma unroll
                            for (int v = 0; v < CPT / 16; ++v) {
                                const int q0 = cb + hf * (CPT / 2) + v * 8;                 // first of 8 queries
                                uint8_t* dst = sDs + (q0 >> 6) * kBoxBytes + r * 128 + ((((q0 & 63) >> 3) ^ (r & 7)) << 4);
                                *reinterpret_cast<uint4*>(dst) = make_uint4(pk[4 * v], pk[4 * v + 1], pk[4 * v + 2], pk[4 * v + 3]);
                            }
                        }
                    }
                }
                if (FUSED) fence_proxy_async_smem();
                tmem_wait_st();
                if (PREC == 2 && DS && a.ds_staged && !summing) mbar_arrive_read_done(&bars[Cfg::kBiasEmpty]);     // (written, here)
            }
#undef PF
#undef PSET
            tc_fence_before_sync();
            mbar_arrive_warp(&bars[b_ready]);
            if (DS && it == sum_steps - 1) {
                // the row's four threads put their sums together, in a fixed order.  They meet before the first sum is left,
                // too: the sums' room is where the rows' -lse and -delta were brought to, and with one key tile nothing else
                // lies between a warp that is here and one that has not read them yet.
                uint32_t meet = 0u;                          // four times a block: every block finds the first parity again
                auto all_met = [&] {
                    mbar_arrive_warp(&bars[Cfg::kSums]);
                    const bool good = mbar_wait(&bars[Cfg::kSums], meet & 1u, abort_flag);
                    ++meet;
                    return __all_sync(0xffffffffu, good);
                };
                auto row_sum = [&](uint64_t mine, float& out) {
                    float x0, x1;
                    f2_unpack(mine, x0, x1);
                    sVec[wg * 128 + r] = x0 + x1;
                    if (!all_met()) return false;
                    out = (sVec[r] + sVec[128 + r]) + (sVec[256 + r] + sVec[384 + r]);
                    return true;
                };
                float sum_p = 0.f, sum_pd = 0.f;
                ok = all_met() && row_sum(sum_p2, sum_p) && all_met() && row_sum(sum_pd2, sum_pd);
                if (!ok) break;
                mbar_arrive_read_done(&bars[Cfg::kRowEmpty]);
                // a row without a result, or one whose lse has lost its sum (all of it masked with a lowest value),
                // keeps what it has
                if (sum_p > 0.f && fabsf(sum_pd) < INFINITY) my_ndelta = -sum_pd / sum_p;
                const float unit = p_mul / sum_p;
                if (fabsf(unit - 1.f) < 0.25f) p_mul *= unit;
            }
            }
            if (KS) mbar_arrive_warp(&bars[Cfg::kVEmpty + (g & 1)]);      // this step's lse / delta rows are read
            prev_tile = strm_tile; prev_head = head_q;
            if (++qi == n_per_head) { qi = 0; ++hg; }
        }

        if (FUSED && n_iter > 0 && ok) ok = drain_dq(g - 1, prev_tile, prev_head);

        if (ROW_MAX) sc_row = sc;
        }
        // ---- epilogue: accumulators -> 16-bit -> swizzled staging -> TMA store.  dK or dQ goes to the place of the block's
        // last U tile, dV to that of its last W tile; warp 19 sends them off and gives the places back to the producer.
        // (Straight from registers a warp's 16-byte stores go to 32 rows each: 2200 cycles at D = 64, 4000 at D = 128.)
        if (ok) ok = item_there((int)((count + 1u) & 3u));
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        // (read again: what is not held through the steps leaves their loop its registers)
        const volatile BwdItem* m = sched + (count & 1u);
        const int n_iter = m->n_iter;
        if (XY_CONV && sched[(count & 1u) ^ 1u].n_iter > 0) ok = convert_xy(0, ((count >> 2) & 1u) ^ (n_iter > 0 ? 1u : 0u));
        const BwdScales sc = ROW_MAX ? sc_row : scales(m);
        if (n_iter > 0 && ok) ok = mbar_wait(&bars[Cfg::kAccDone], (count >> 2) & 1u, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        constexpr int kCols = D / NWG;                     // my share of the D accumulator columns: 16 or 32
        constexpr int kOuts = (KS) ? 2 : 1;
        if (n_iter > 0) {
#pragma unroll
            for (int o = 0; o < kOuts; ++o) {
                const uint32_t tacc = (o == 0 ? tAcc1 : tAcc2) + lane_off + (uint32_t)(wg * kCols);
                const float mul = (o == 0) ? sc.acc1_mul : sc.acc2_mul;
                uint8_t* stage = o == 0 ? sU + ((g - 1) % UST) * TILE : sW + ((g - 1) % WST) * TILE;
                uint32_t acc[kCols];
                if constexpr (kCols == 32) tmem_ld_32x32(tacc, acc);
                else                       tmem_ld_32x16(tacc, acc);
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < kCols / 8; ++q) {
                    uint4 v4;
                    v4.x = pack2<BF16>(__uint_as_float(acc[q * 8 + 0]) * mul, __uint_as_float(acc[q * 8 + 1]) * mul);
                    v4.y = pack2<BF16>(__uint_as_float(acc[q * 8 + 2]) * mul, __uint_as_float(acc[q * 8 + 3]) * mul);
                    v4.z = pack2<BF16>(__uint_as_float(acc[q * 8 + 4]) * mul, __uint_as_float(acc[q * 8 + 5]) * mul);
                    v4.w = pack2<BF16>(__uint_as_float(acc[q * 8 + 6]) * mul, __uint_as_float(acc[q * 8 + 7]) * mul);
                    const int col = wg * kCols + q * 8;
                    *reinterpret_cast<uint4*>(stage + (col >> 6) * kBoxBytes + r * 128 + ((((col & 63) >> 3) ^ (r & 7)) << 4)) = v4;
                }
            }
            tc_fence_before_sync();                        // (the next block's first hand-off lets them be overwritten)
            fence_proxy_async_smem();
            mbar_arrive_warp(&bars[Cfg::kEpi]);
        } else if (m->tile * kTile + r < (KS ? a.Nk : a.Nq)) {
            // no query sees this key tile
            const int64_t row = m->tile * kTile + r;
            uint16_t* dst1 = (uint16_t*)a.out1 + m->b * a.o1_sb + row * a.o1_sn + m->head_x * a.o1_sh;
            uint16_t* dst2 = (uint16_t*)a.out2 + m->b * a.o2_sb + row * a.o2_sn + m->head_x * a.o2_sh;
#pragma unroll
            for (int col = wg * kCols; col < (wg + 1) * kCols; col += 8) {
                if (PREC != 0 && col >= a.d) break;
                *reinterpret_cast<uint4*>(dst1 + col) = make_uint4(0u, 0u, 0u, 0u);
                if (KS) *reinterpret_cast<uint4*>(dst2 + col) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        mbar_arrive_warp(&bars[Cfg::kSchedEmpty + (count & 1u)]);
        count = ((count + 1u) & 3u) | ((count & 4u) ^ (n_iter > 0 ? 4u : 0u));
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0 && *abort_flag) report_status(a.status, 2 + MODE);
    // the end of this grid must still mean the end of the dK/dV grid before it in the stream
    if (MODE == 1) grid_dependency_wait();
}

// Block-wide maximum of absmax16_acc's patterns, as a float, folded into *slot (an fp32 bit pattern; for
// non-negative floats the unsigned order is the numeric order, so atomicMax on the bits is exact).
template <typename T>
__device__ __forceinline__ void absmax16_commit(uint32_t m, float* slot, uint32_t* red) {
    m = max(m & 0xFFFFu, m >> 16);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = max(m, red[w]);
        const unsigned short bits = (unsigned short)m;
        const float f = to_f32<T>(*reinterpret_cast<const T*>(&bits));
        atomicMax(reinterpret_cast<uint32_t*>(slot), __float_as_uint(f));
    }
}

// Preprocess launch.  Blocks [0, n_row_blocks): negated delta and the shifted, negated, scaled lse (the
// main kernels add them), and max |dO| of the block's column.  D / 8 lanes share one (b, h, padded query
// row), 16 bytes of O and dO each, so a warp covers 256 / D rows; a block's rows lie in one (b, h).
// Blocks beyond: max |V| over a slab of one (b, K/V head) column's visible keys.
// ranges[(b * Hkv + hk) * 2 + {0, 1}] = max |dO| over the K/V head's query heads, max |V|; zeroed before.
// COPIES (bf16): also the fp16 copies the main kernels stream, dense (B, Nq, H, D): Q as it is, dO row
// by row normalised to max < 2^15 by 2^-e_i, with e_i kept in `erow` and folded into the two vectors
// (lse' = kPShift - lse*log2(e) + e_i, -delta * 2^-e_i: the "row form" of make_scales).
struct PreprocessCopies {
    const void* o_lo; int64_t l_sb, l_sn, l_sh;     // optional residual of O (any dtype)
    const void* q; int64_t q_sb, q_sn, q_sh;
    uint16_t* q16; uint16_t* do16; float* erow;
    int pairs;                                      // PREC != 0: -lse instead of kPShift - lse*log2(e), maxima of finite values
};
// A head size below D (pair instances) leaves the lanes beyond it idle.
template <typename T, int D, bool COPIES>
__global__ void __launch_bounds__(256)
bwd_preprocess_kernel(int d, const T* __restrict__ o, const T* __restrict__ d_o, const float* __restrict__ lse,
                      float* __restrict__ lse2, float* __restrict__ delta, float* __restrict__ ranges,
                      int B, int Nq, int H, int Hkv, int nq_pad,
                      int64_t o_sb, int64_t o_sn, int64_t o_sh, int64_t g_sb, int64_t g_sn, int64_t g_sh,
                      const T* __restrict__ v, int64_t v_sb, int64_t v_sn, int64_t v_sh, int Nk,
                      const int32_t* __restrict__ kv_len, int n_row_blocks, int v_slabs, const PreprocessCopies cp) {
    grid_launch_dependents();                  // the dK/dV kernel, which waits for this grid's end
    constexpr int LPR = D / 8;                 // lanes per row
    constexpr int RPW = 32 / LPR;              // rows per warp
    constexpr int kVRows = 256;                // keys per slab of the V scan
    __shared__ uint32_t red[8];
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    if ((int)blockIdx.x >= n_row_blocks) {
        const int vb = (int)blockIdx.x - n_row_blocks;
        const int slab = vb % v_slabs, col = vb / v_slabs;          // col = b * Hkv + hk
        const int hk = col % Hkv, b = col / Hkv;
        const int nk = kv_len_of(kv_len, b, Nk);
        uint32_t m = 0u;
        const int j_end = min(nk, (slab + 1) * kVRows);
        for (int j = slab * kVRows + (int)(threadIdx.x / LPR); j < j_end && sub * 8 < d; j += 256 / LPR)
        {
            const uint4 piece = *reinterpret_cast<const uint4*>(v + b * v_sb + (int64_t)j * v_sn + hk * v_sh + sub * 8);
            if (!cp.pairs) { m = absmax16_acc(m, piece); continue; }
            const uint32_t mp = finite_piece<T>(absmax16_acc(0u, piece));
            asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(mp));
        }
        absmax16_commit<T>(m, ranges + 2 * (int64_t)col + 1, red);
        return;
    }
    // a block takes one 128-row tile of one (b, h): kPasses passes of 256 / LPR rows, a pass's loads
    // issued together; one reduction of max |dO| per block
    constexpr int kRowsPerPass = 8 * RPW;
    constexpr int kPasses = 128 / kRowsPerPass;
    const int tiles_per_col = nq_pad / 128;
    const int64_t bh = (int64_t)blockIdx.x / tiles_per_col;
    const int i0 = ((int)blockIdx.x - (int)(bh * tiles_per_col)) * 128 + (int)(threadIdx.x >> 5) * RPW + lane / LPR;
    const int h = (int)(bh % H), b = (int)(bh / H);
    const T* op = o + b * o_sb + h * o_sh + sub * 8;
    const T* gp = d_o + b * g_sb + h * g_sh + sub * 8;
    const T* lp = cp.o_lo ? reinterpret_cast<const T*>(cp.o_lo) + b * cp.l_sb + h * cp.l_sh + sub * 8 : nullptr;
    const T* qp = COPIES ? reinterpret_cast<const T*>(cp.q) + b * cp.q_sb + h * cp.q_sh + sub * 8 : nullptr;
    uint32_t m = 0u;
    constexpr int kTogether = COPIES ? 2 : 4;                  // passes whose loads are in flight together
#pragma unroll kTogether
    for (int ps = 0; ps < kPasses; ++ps) {
        const int i = i0 + ps * kRowsPerPass;
        const int64_t row = bh * nq_pad + i;
        const bool in = i < Nq;
        uint4 vo = make_uint4(0, 0, 0, 0), vg = vo, vl = vo, vq = vo;
        const float lse_i = in && sub == 0 ? lse[bh * Nq + i] : 0.f;
        if (in && sub * 8 < d) {
            vo = *reinterpret_cast<const uint4*>(op + (int64_t)i * o_sn);
            vg = *reinterpret_cast<const uint4*>(gp + (int64_t)i * g_sn);
            if (lp) vl = *reinterpret_cast<const uint4*>(lp + (int64_t)i * cp.l_sn);
            if (COPIES) vq = *reinterpret_cast<const uint4*>(qp + (int64_t)i * cp.q_sn);
        }
        const T* eo = reinterpret_cast<const T*>(&vo);
        const T* eg = reinterpret_cast<const T*>(&vg);
        const T* el = reinterpret_cast<const T*>(&vl);
        float s = 0.f;
        // delta from the output as the forward computed it (o + o_lo) when the residual is there
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(to_f32<T>(eo[e]) + to_f32<T>(el[e]), to_f32<T>(eg[e]), s);
#pragma unroll
        for (int off = LPR / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        uint32_t m_mine = absmax16_acc(0u, vg);
        if (cp.pairs) m_mine = finite_piece<T>(m_mine);
        m = max(m, max(m_mine & 0xFFFFu, m_mine >> 16));
        int e_i = 0;
        if (COPIES) {
            // the row's largest |dO| (a bf16 bit pattern) over the lanes that share the row
            uint32_t mr = max(m_mine & 0xFFFFu, m_mine >> 16);
#pragma unroll
            for (int off = LPR / 2; off > 0; off >>= 1) mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, off));
            e_i = log2_bound_bits(mr << 16) - 15;
            if (in) {
                const int64_t at = (((int64_t)b * Nq + i) * H + h) * D + sub * 8;
                const uint64_t mul2 = f2_pack(pow2i(-e_i), pow2i(-e_i));
                *reinterpret_cast<uint4*>(cp.q16 + at) = make_uint4(bf16x2_to_f16x2(vq.x), bf16x2_to_f16x2(vq.y),
                                                                    bf16x2_to_f16x2(vq.z), bf16x2_to_f16x2(vq.w));
                *reinterpret_cast<uint4*>(cp.do16 + at) = make_uint4(bf16x2_to_f16x2(vg.x, mul2), bf16x2_to_f16x2(vg.y, mul2),
                                                                     bf16x2_to_f16x2(vg.z, mul2), bf16x2_to_f16x2(vg.w, mul2));
            }
        }
        if (sub == 0) {
            if (in) { delta[row] = -s * pow2i(-e_i); lse2[row] = cp.pairs ? -lse_i : kPShift - lse_i * kLog2e + (float)e_i; }
            else    { delta[row] = 0.f; lse2[row] = -INFINITY; }
            if (COPIES) cp.erow[row] = in ? (float)e_i : 0.f;
        }
    }
    const int group = H / Hkv;
    absmax16_commit<T>(m, ranges + 2 * ((int64_t)b * Hkv + h / group), red);
}

// fused backward: fp32 dQ sums (tiles of [D/4][128 rows][4]) * scale -> dQ in the call's dtype and layout
template <typename T, int D>
__global__ void __launch_bounds__(256)
bwd_dq_convert_kernel(const float* __restrict__ acc, T* __restrict__ dq, int Nq, int H, int n_tiles, float scale_in,
                      int64_t sb, int64_t sn, int64_t sh, const float* __restrict__ ranges, int Hkv, float inv_keep) {
    const int tile = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    // the sums carry the column's dS scaling (see "number formats"): the same constant the dK epilogue uses
    const float scale = make_scales(ranges + 2 * ((int64_t)b * Hkv + h / (H / Hkv)), D, inv_keep, scale_in,
                                    kDoAsIs).acc1_mul;     // acc1_mul does not depend on dO's form
    const float* src = acc + (((int64_t)b * H + h) * n_tiles + tile) * (int64_t)(kTile * D);
    const int row = threadIdx.x & 127;
    const int i = tile * kTile + row;
    if (i >= Nq) return;
    T* out = dq + b * sb + (int64_t)i * sn + h * sh;
#pragma unroll
    for (int cg = threadIdx.x >> 7; cg < D / 8; cg += 2) {      // 8 columns = two 4-column groups
        const float4 lo = *reinterpret_cast<const float4*>(src + ((int64_t)(2 * cg) * kTile + row) * 4);
        const float4 hi = *reinterpret_cast<const float4*>(src + ((int64_t)(2 * cg + 1) * kTile + row) * 4);
        uint4 v4;
        v4.x = pack2<std::is_same<T, __nv_bfloat16>::value>(lo.x * scale, lo.y * scale);
        v4.y = pack2<std::is_same<T, __nv_bfloat16>::value>(lo.z * scale, lo.w * scale);
        v4.z = pack2<std::is_same<T, __nv_bfloat16>::value>(hi.x * scale, hi.y * scale);
        v4.w = pack2<std::is_same<T, __nv_bfloat16>::value>(hi.z * scale, hi.w * scale);
        *reinterpret_cast<uint4*>(out + cg * 8) = v4;
    }
}

// INLINE: bf16 call without room for the fp16 copies (the workspace-free entry point): the main kernels
// convert their tiles themselves.
// the kernel instance and its shared memory for a dropout form (0 none, 1 drawn in the kernel, 2 loaded;
// the converting-in-kernel instances, which serve the entry without a workspace, never load)
template <int D, bool BF16, int MODE, bool INLINE, int PREC, bool DS = false>
auto pick_kernel(int drop) {
    if (drop == 2 && !INLINE) return bwd_sm100_kernel<D, BF16, MODE, kNWG, INLINE ? 1 : 2, INLINE, PREC, DS>;
    if constexpr (PREC == 2) return bwd_sm100_kernel<D, BF16, MODE, kNWG, 0, INLINE, PREC, DS>;       // bias_is_staged(): never drop = 1
    else return drop ? bwd_sm100_kernel<D, BF16, MODE, kNWG, 1, INLINE, PREC, DS> : bwd_sm100_kernel<D, BF16, MODE, kNWG, 0, INLINE, PREC, DS>;
}
template <int D, int MODE, int PREC>
int pick_smem(int drop) {
    if constexpr (PREC == 2) return drop ? BwdCfg<D, MODE, 2, PREC>::kSmemBytes : BwdCfg<D, MODE, 0, PREC>::kSmemBytes;
    else return drop == 2 ? BwdCfg<D, MODE, 2, PREC>::kSmemBytes
                     : (drop ? BwdCfg<D, MODE, 1, PREC>::kSmemBytes : BwdCfg<D, MODE, 0, PREC>::kSmemBytes);
}

template <int D, bool BF16, bool INLINE, int PREC>
int launch(const fa_b200_params& p, const BwdWorkspace& ws) {
    using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    const CUtensorMapDataType dt = BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    constexpr bool COPIES = BF16 && !INLINE && PREC == 0;
    cudaStream_t st = (cudaStream_t)p.stream;
    const int nq_pad = (int)align_up((size_t)p.Nq, 128);
    char* wsp = (char*)p.workspace;
    float* delta = (float*)(wsp + ws.delta_off);
    float* lse2 = (float*)(wsp + ws.lse2_off);
    float* ranges = (float*)(wsp + ws.rng_off);
    if (COPIES && (ws.q16_bytes == 0 || ws.do16_bytes == 0)) { set_error("workspace layout lacks the fp16 copies"); return FA_EWORKSPACE; }

    const bool fused = ws.dq_bytes > 0;
    float* dq_acc = fused ? (float*)(wsp + ws.dq_off) : nullptr;
    // dropout: 0 none, 1 the kernels draw their bits, 2 they load them from the call's bit buffer
    int drop = dropout_threshold(p.dropout_p) != 0u ? 1 : 0;
    const size_t bits_one = dropout_bits_bytes(p);
    if (!INLINE && drop && p.dropout_bits && p.dropout_bits_bytes >= 2 * bits_one) drop = 2;

    const int phases = p.bwd_phases ? p.bwd_phases : 7;
    if (phases & 1) {
        if (fused) FA_CUDA_CHECK(cudaMemsetAsync(dq_acc, 0, ws.dq_bytes, st));
        FA_CUDA_CHECK(cudaMemsetAsync(ranges, 0, ws.rng_bytes, st));
        const int64_t n_row_blocks64 = (int64_t)p.B * p.H * (nq_pad / 128);      // one block per 128-row tile
        const int v_slabs = (p.Nk + 255) / 256;
        const int64_t n_blocks = n_row_blocks64 + (int64_t)p.B * p.Hkv * v_slabs;
        if (n_blocks > 0x7fffffff) { set_error("problem too large for the preprocess grid"); return FA_EUNSUPPORTED; }
        const int n_row_blocks = (int)n_row_blocks64;
        PreprocessCopies cp = {};
        cp.pairs = PREC != 0;
        cp.o_lo = p.o_lo.ptr; cp.l_sb = p.o_lo.stride_b; cp.l_sn = p.o_lo.stride_n; cp.l_sh = p.o_lo.stride_h;
        if (COPIES) {
            cp.q = p.q.ptr; cp.q_sb = p.q.stride_b; cp.q_sn = p.q.stride_n; cp.q_sh = p.q.stride_h;
            cp.q16 = (uint16_t*)(wsp + ws.q16_off); cp.do16 = (uint16_t*)(wsp + ws.do16_off);
            cp.erow = (float*)(wsp + ws.erow_off);
        }
        bwd_preprocess_kernel<T, D, COPIES><<<(unsigned)n_blocks, 256, 0, st>>>(
            p.D, (const T*)p.o.ptr, (const T*)p.d_o.ptr, p.lse, lse2, delta, ranges, p.B, p.Nq, p.H, p.Hkv, nq_pad,
            p.o.stride_b, p.o.stride_n, p.o.stride_h, p.d_o.stride_b, p.d_o.stride_n, p.d_o.stride_h,
            (const T*)p.v.ptr, p.v.stride_b, p.v.stride_n, p.v.stride_h, p.Nk, p.kv_lengths, n_row_blocks, v_slabs, cp);
        FA_CUDA_CHECK(cudaGetLastError());
    }

    CUtensorMap mq, mk, mv, mg, mdq, mdk, mdv, mq16, mg16, mk16;
    int r;
    auto mk_map = [&](CUtensorMap* m, const fa_b200_tensor& t, int N, int H) {
        return cached_tmap_bnhd(m, t.ptr, dt, 2, p.B, N, H, p.D, t.stride_b, t.stride_n, t.stride_h, 128, 64, true);
    };
    // a dense fp16 (B, N, H, D) copy in the workspace
    auto mk_copy = [&](CUtensorMap* m, size_t off, int N, int H) {
        return cached_tmap_bnhd(m, wsp + off, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.B, N, H, D, (int64_t)N * H * D,
                                (int64_t)H * D, (int64_t)D, 128, 64, true);
    };
    if ((r = mk_map(&mq, p.q, p.Nq, p.H)) || (r = mk_map(&mk, p.k, p.Nk, p.Hkv)) ||
        (r = mk_map(&mv, p.v, p.Nk, p.Hkv)) || (r = mk_map(&mg, p.d_o, p.Nq, p.H)) ||
        (r = mk_map(&mdq, p.dq, p.Nq, p.H)) || (r = mk_map(&mdk, p.dk, p.Nk, p.Hkv)) ||
        (r = mk_map(&mdv, p.dv, p.Nk, p.Hkv))) {
        set_error("cuTensorMapEncodeTiled failed (%d)", r);
        return FA_ECUDA;
    }
    mq16 = mq; mg16 = mg; mk16 = mk;
    if (COPIES) {
        if ((r = mk_copy(&mq16, ws.q16_off, p.Nq, p.H)) || (r = mk_copy(&mg16, ws.do16_off, p.Nq, p.H)) ||
            (ws.k16_bytes && (r = mk_copy(&mk16, ws.k16_off, p.Nk, p.Hkv)))) {
            set_error("cuTensorMapEncodeTiled failed (%d)", r);
            return FA_ECUDA;
        }
    }
    CUtensorMap mb = mq, mds = mq;
    BwdArgs a;
    a.bias_b = p.bias.stride_b != 0 && p.B > 1; a.bias_h = p.bias.stride_h != 0 && p.H > 1;
    if (PREC == 2 && (r = cached_tmap_bnhd(&mb, p.bias.ptr, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.bias_b ? p.B : 1, p.Nq, a.bias_h ? p.H : 1,
                                           p.Nk, p.bias.stride_b, p.bias.stride_n, p.bias.stride_h, 128, 32, 1))) {
        set_error("cuTensorMapEncodeTiled failed for the bias (%d)", r);
        return FA_ECUDA;
    }
    a.ds_staged = PREC == 2 && p.d_scores && p.Nk % 4 == 0 && ((uintptr_t)p.d_scores & 15u) == 0;
    if (a.ds_staged && (r = cached_tmap_bnhd(&mds, p.d_scores, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p.B, p.Nq, p.H, p.Nk,
                                             (int64_t)p.H * p.Nq * p.Nk, p.Nk, (int64_t)p.Nq * p.Nk, 128, 32, 1))) {
        set_error("cuTensorMapEncodeTiled failed for d_scores (%d)", r);
        return FA_ECUDA;
    }
    a.lse2 = lse2; a.delta = delta; a.ranges = ranges; a.dq_acc = dq_acc; a.status = p.status_word; a.wait_limit_ms = p.wait_limit_ms;
    a.erow = COPIES ? (const float*)(wsp + ws.erow_off) : nullptr;
    a.kv_len = p.kv_lengths;
    a.B = p.B; a.Nq = p.Nq; a.Nk = p.Nk; a.H = p.H; a.Hkv = p.Hkv; a.nq_pad = nq_pad;
    {
        // columns whose Q, K, V and dO (16-bit) fit the budget
        const int64_t col_bytes = 2 * ((int64_t)p.Nq + p.Nk) * D * 2;
        const int64_t g = (int64_t)tile::kBwdGroupBytes / (col_bytes > 0 ? col_bytes : 1);
        a.cols_per_group = (int)(g < 1 ? 1 : (g > 65535 ? 65535 : g));
    }
    a.group = p.H / p.Hkv;
    a.causal = p.causal;
    a.shift = p.causal ? p.causal_shift : 0;
    a.scale = p.scale;
    a.scale_log2 = p.scale * kLog2e;
    a.score_scale = pair_score_scale(p);
    a.dp_gain = 1.f + pair_truncation(p);
    a.drop_thr = dropout_threshold(p.dropout_p);
    a.inv_keep = 1.f / (1.f - dropout_effective_p(p.dropout_p));
    a.key = philox_make_key(p.seed, p.offset);
    a.rng = dropout_origin_of(p);
    a.bits_q = (const uint4*)p.dropout_bits;
    a.bits_k = (const uint32_t*)((const char*)p.dropout_bits + bits_one);
    a.nk_pad = (int)align_up((size_t)p.Nk, 128);
    a.d = p.D;
    a.bias = (const float*)p.bias.ptr;
    a.bias_sb = p.bias.stride_b; a.bias_sn = p.bias.stride_n; a.bias_sh = p.bias.stride_h;
    a.bias_vec = (((uintptr_t)p.bias.ptr & 15u) == 0 && (p.bias.stride_b | p.bias.stride_n | p.bias.stride_h) % 4 == 0) ? 1 : 0;
    a.d_scores = p.d_scores;
    a.ds_vec = (p.Nk % 4 == 0 && ((uintptr_t)p.d_scores & 15u) == 0) ? 1 : 0;
    if (drop == 2 && !p.dropout_bits_ready && (phases & 1)) {
        int rc = launch_dropout_bits(p, (void*)a.bits_q, (void*)a.bits_k);
        if (rc) return rc;
    }

    auto outputs = [&](const fa_b200_tensor& t1, const fa_b200_tensor& t2) {
        a.out1 = t1.ptr; a.o1_sb = t1.stride_b; a.o1_sn = t1.stride_n; a.o1_sh = t1.stride_h;
        a.out2 = t2.ptr; a.o2_sb = t2.stride_b; a.o2_sn = t2.stride_n; a.o2_sh = t2.stride_h;
    };
    static std::mutex smem_mu;             // per (D, dtype, INLINE) instance of this function
    static uint64_t smem_done[9] = {};     // [kernel mode x dropout form] -> devices whose limit is set
    constexpr int kThreads = 128 * kNWG + kExtraThreads;
    const dim3 grid_kv((p.Nk + kTile - 1) / kTile, p.Hkv, p.B);
    const dim3 grid_q((p.Nq + kTile - 1) / kTile, p.H, p.B);
    if constexpr (D == 64 && PREC == 0) if (fused) {
        // one key-stationary kernel for dK, dV and the fp32 dQ sums, then the conversion of dQ
        auto k2 = pick_kernel<D, BF16, 2, INLINE, PREC>(drop);
        const int smem2 = pick_smem<D, 2, PREC>(drop);
        FA_CUDA_CHECK(set_smem_limit_once(k2, smem2, p.device, &smem_done[6 + drop], &smem_mu));
        if (phases & 2) {
            outputs(p.dk, p.dv);
            k2<<<grid_kv, kThreads, smem2, st>>>(mk, mv, mq16, mg16, mdk, mdv, mdk, mb, mds, a);
            FA_CUDA_CHECK(cudaGetLastError());
        }
        if (phases & 4) {
            bwd_dq_convert_kernel<T, D><<<grid_q, 256, 0, st>>>(dq_acc, (T*)p.dq.ptr, p.Nq, p.H, nq_pad / kTile, p.scale,
                                                               p.dq.stride_b, p.dq.stride_n, p.dq.stride_h, ranges, p.Hkv,
                                                               a.inv_keep);
            FA_CUDA_CHECK(cudaGetLastError());
        }
        return FA_OK;
    }
    if (COPIES && ws.k16_bytes == 0) { set_error("workspace layout lacks the fp16 copy of K"); return FA_EWORKSPACE; }
    auto k0 = pick_kernel<D, BF16, 0, INLINE, PREC>(drop);
    auto k1 = pick_kernel<D, BF16, 1, INLINE, PREC>(drop);
    if constexpr (PREC != 0) if (p.d_scores) k1 = pick_kernel<D, BF16, 1, INLINE, PREC, true>(drop);
    const int smem0 = pick_smem<D, 0, PREC>(drop), smem1 = pick_smem<D, 1, PREC>(drop);
    FA_CUDA_CHECK(set_smem_limit_once(k0, smem0, p.device, &smem_done[drop], &smem_mu));
    FA_CUDA_CHECK(set_smem_limit_once(k1, smem1, p.device, &smem_done[(PREC && p.d_scores ? 6 : 3) + drop], &smem_mu));
    if (phases & 2) {
        // stationary K_j, V_j; streamed Q_i, dO_i (bf16 with copies: their fp16 copies; the kernel leaves
        // the fp16 copy of K behind for the dQ kernel)
        outputs(p.dk, p.dv);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid_kv; cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = smem0; cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = (phases & 1) ? 1 : 0;        // only behind the preprocess launch of this call
        FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k0, mk, mv, mq16, mg16, mdk, mdv, mk16, mb, mds, a));
    }
    if (phases & 4) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid_q; cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = smem1; cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        // Only behind the dK/dV kernel of this call, and only while one head's K and V are small
        // beside L2 (the two kernels stream different heads' tiles at the same time): measured on
        // B200 (H32 D128 causal) the overlap takes 1 % off the backward at N = 4096; longer
        // sequences showed no gain.  Never with the fp16 copies: the dQ kernel streams the copy of K
        // that the dK/dV kernel is still writing.
        cfg.numAttrs = (!COPIES && (phases & 2) && (int64_t)p.Nk * D * 4 <= (int64_t)tile::kBwdOverlapMaxKvBytes) ? 1 : 0;
        // stationary Q_i (its fp16 copy), dO_i; streamed K_j (its fp16 copy), V_j
        outputs(p.dq, p.dq);
        FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k1, mq16, mg, mk16, mv, mdq, mdq, mdq, mb, mds, a));
    }
    return FA_OK;
}

}  // namespace

#ifndef FA_PAIR_INSTANCES
bool sm100_bwd_fused_supported(const fa_b200_params& p) {
    // D = 64 only.  At D = 128 tensor memory is full (S^T, dP^T, dK, dV), the per-step dQ tile has
    // to share dP^T's columns, which serialises the step, and the fp32 additions (64 KB per step)
    // cost more than recomputing S and dP in a second kernel: measured on B200 (B4 N4096 H32
    // causal) 2.12 ms against 1.95 ms for the two kernels.
    return tile::bwd_one_kernel(p.D);
}

int sm100_bwd(const fa_b200_params& p, const BwdWorkspace& ws) {
    if (p.dtype == FA_B200_BF16) {
        if (ws.q16_bytes == 0) return p.D == 128 ? launch<128, true, true, 0>(p, ws) : launch<64, true, true, 0>(p, ws);
        return p.D == 128 ? launch<128, true, false, 0>(p, ws) : launch<64, true, false, 0>(p, ws);
    }
    return p.D == 128 ? launch<128, false, false, 0>(p, ws) : launch<64, false, false, 0>(p, ws);
}

#else
int sm100_pair_bwd(const fa_b200_params& p, const BwdWorkspace& ws) {
    if (bias_is_staged(p, 2 * dropout_bits_bytes(p))) {
        if (p.dtype == FA_B200_BF16) return p.D > 64 ? launch<128, true, false, 2>(p, ws) : launch<64, true, false, 2>(p, ws);
        return p.D > 64 ? launch<128, false, false, 2>(p, ws) : launch<64, false, false, 2>(p, ws);
    }
    if (p.dtype == FA_B200_BF16) return p.D > 64 ? launch<128, true, false, 1>(p, ws) : launch<64, true, false, 1>(p, ws);
    return p.D > 64 ? launch<128, false, false, 1>(p, ws) : launch<64, false, false, 1>(p, ws);
}
#endif

}  // namespace fa
