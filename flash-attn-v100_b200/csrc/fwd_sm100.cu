// Attention forward for sm_100a: TMA -> shared memory -> tcgen05.mma with
// accumulators in tensor memory, warp-specialised, persistent.
//
// Replaces the reference's Triton forward kernel
// (kernels/forward_kernel.py:18-243) and its launcher (:246-387).
//
// Work: a "pair" is two consecutive 128-row query tiles of one (batch, head);
// it walks the key/value sequence in 128-row blocks.  The grid is one CTA per
// SM; CTA c processes work items c, c + grid, c + 2 grid, ...  Under a causal
// mask an item is a pair together with its mirror (pair p and pair P-1-p), so
// that every item costs the same number of key blocks and a static round-robin
// is balanced; items of one head are adjacent, so the CTAs running at any time
// share a few heads' K/V in L2.  Nothing is re-initialised between pairs: the
// K/V ring, the barriers' phases and tensor memory carry on, and the next
// pair's Q and first K/V blocks are loaded while the current pair drains.
//
//   warp 9      TMA producer: Q tiles per pair, K_j / V_j into two rings
//   warp 8      MMA issuer (one elected thread):
//                   S_t = Q_t K_j^T          (SS MMA, both operands K-major)
//                   O_t += P_t V_j           (TS MMA: P_t from TMEM, V_j MN-major)
//               issue order  S0(0) S1(0) | PV0(j) S0(j+1) PV1(j) S1(j+1) ...
//               so that the softmax of one tile overlaps the MMAs of the other; each PV
//               is issued in two 64-key halves, the first as soon as that half of P_t
//               is in TMEM (the threads are still computing the second)
//   warps 0-3   softmax + epilogue of tile 0, one thread per query row (TMEM lane)
//   warps 4-7   softmax + epilogue of tile 1
//   warps 10-11 bf16 inputs: convert each V_j tile to fp16 in place as it lands, so that PV runs
//               f16 x f16 with P rounded to fp16 instead of bf16 (see sm100_ptx.cuh); fp16 inputs: idle
//               (the two warps complete the third warpgroup for setmaxnreg)
//
// Online softmax in the log2 domain with scale*log2(e) folded into one FMA (pair instances: in natural units, see there).
// The running maximum is only refreshed when it grows by more than 2^8 (warp
// vote), so the O accumulator in TMEM is rescaled rarely; the final division
// by the row sum makes the result exact either way.  P is rounded to fp16 (whatever
// the input dtype) and written over S in TMEM; dropout zeroes P entries (the 1/(1-p)
// factor is applied once to O), the row sum uses the undropped P.
//
// TMEM columns: S0/P0 [0,128)  S1/P1 [128,256)  O0 [256,256+D)  O1 [384,384+D).
// O_t of the next pair is first written by a PV MMA that waits for P_t, which
// the owning threads produce only after their epilogue has read O_t.
//
// Every mbarrier wait is bounded; on a time-out the CTA raises its abort flag,
// every role unwinds, TMEM is freed and the status word is set.
#include "fa_common.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"
#include "tile_config.cuh"
#include <type_traits>

namespace fa {
namespace {

using namespace ptx;

constexpr int kBlockM = tile::kBlockM;      // query rows per tile
constexpr int kBlockN = tile::kBlockN;      // key rows per block
constexpr int kThreads = 32 * tile::kFwdWarps;   // 2 softmax warpgroups + 1 warpgroup holding the MMA, TMA and converting warps
constexpr int kBoxBytes = 128 * 128;   // one TMA box: 128 rows x 64 16-bit elements
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = tile::kFwdRescaleLog2;   // log2 units
// The first 64 keys of P are handed to the MMA warp after this many of the second half's 64
// exponentials (a multiple of 4), when their tcgen05.st has had time to complete.
constexpr int kHalfSignalAt = tile::kFwdHalfSignalAt;
// Register split after setmaxnreg.  The pool is what the CTA was launched with, 168 registers for
// each of its 384 threads, not the whole file: a split that asks for more makes
// setmaxnreg.inc wait for ever.
constexpr int kRegsSoftmax = tile::kFwdRegsSoftmax, kRegsOther = tile::kFwdRegsOther;
static_assert(256 * kRegsSoftmax + 128 * kRegsOther <= 168 * kThreads, "register split exceeds the CTA's allocation");
static_assert(tile::kFwdQTilesPerCta == 2, "the kernel is written for two query tiles per work item");

// PREC: how P and the operands reach the MMAs.
//   0  fp16 / bf16 calls with D = 64 or 128: P as one fp16 value (kernel comment above)
//   1  "pair": 16-bit calls with an additive bias or another head size (any multiple of 8 up to 128; the
//      tiles are padded to 64 or 128 columns by TMA's zero fill, the MMA K-steps and N stop at the head
//      size).  P is handed over as hi + lo in the inputs' own format, two MMAs per K-step of P V, so P keeps
//      17 (bf16) or 22 (fp16) significant bits and a bf16 V needs no conversion.
//   2  the same with the bias brought to shared memory by TMA, in chunks of 128 rows x 32 columns: a thread needs 32
//      consecutive values of its own row, and read straight from global memory a warp's load touches 32 lines.
//      Dense or batch / head broadcast biases whose rows TMA can address; one that is broadcast over the queries is
//      the same value for a whole warp and stays with PREC = 1.
// SCHED: how the work is divided (plan_schedule).
//   0  whole pairs of 128-row tiles, round robin (kernel comment above)
//   1  the split schedule, with packed tiles or plain ones
//   2  the same for a call whose rows fit one tile (decoding): the tile's even key blocks go through S_0, P_0 and O_0,
//      the odd ones through S_1, P_1 and O_1, and the two sums are put together in the epilogue; the room of the
//      second query tile goes to the K and V rings.
template <int D, int PREC, int SCHED>
struct FwdCfg {
    static constexpr int kNBox = D / 64;
    static constexpr int kTileBytes = kNBox * kBoxBytes;
    static constexpr int kPolyPeriod = tile::fwd_poly_period(D);
    static constexpr int kQTiles = SCHED == 2 ? 1 : 2;
    static constexpr int kStages = SCHED == 2 ? tile::fwd_one_tile_kv_stages(D)
                                                 : (PREC == 2 ? tile::fwd_bias_kv_stages(D) : tile::fwd_kv_stages(D));
    static constexpr int kBiasSlots = PREC == 2 ? tile::fwd_bias_slots(D) : 0;         // chunks of 16 KB per query tile
    static constexpr int kBiasBytes = 2 * kBiasSlots * kBoxBytes;
    // barrier slots
    static constexpr int kQFull = 0;                       // [2]
    static constexpr int kQEmpty = 2;                      // [2] last S MMA of the pair has read Q_t
    static constexpr int kKFull = 4;                       // [kStages]
    static constexpr int kKEmpty = kKFull + kStages;
    static constexpr int kVFull = kKEmpty + kStages;
    static constexpr int kVEmpty = kVFull + kStages;
    static constexpr int kSFull = kVEmpty + kStages;       // [2]
    static constexpr int kPFull = kSFull + 2;              // [2] one arrival per warp of the warpgroup
    static constexpr int kODone = kPFull + 2;              // [2]
    static constexpr int kPHalf = kODone + 2;              // [2] first 64 keys of P_t stored (one arrival per warp)
    static constexpr int kVConv = kPHalf + 2;              // [kStages] V_j converted to fp16 (one arrival per converting warp)
    static constexpr int kMlFull = kVConv + kStages;       // SCHED = 2: the odd blocks' maxima and sums are in shared memory
    static constexpr int kORead = kMlFull + 1;             // SCHED = 2: O_1 has been read (both: one arrival per warp of a warpgroup)
    static constexpr int kBiasFull = kORead + 1;           // PREC = 2: [2 tiles][kBiasSlots]
    static constexpr int kBiasEmpty = kBiasFull + 2 * kBiasSlots;      // ... one arrival per warp of the warpgroup
    static constexpr int kNumBars = kBiasEmpty + 2 * kBiasSlots;
    static constexpr int kMlBytes = SCHED == 2 ? kBlockM * 8 : 0;
    static constexpr int kWalkBytes = SCHED ? 8 * 40 : 0;  // a WalkRecord per softmax warp
    static constexpr int kSmemBytes = (kQTiles + 2 * kStages) * kTileBytes + kBiasBytes + kNumBars * 8 + 64 + kMlBytes + kWalkBytes + 1024;
    static_assert(kSmemBytes <= 232448, "shared-memory plan does not fit");
};

struct FwdArgs {
    void* o;                       // (B, Nq, H, D) output, element strides below
    int64_t o_sb, o_sn, o_sh;
    void* o_lo;                    // optional residual of the output (what rounding O to 16 bits dropped)
    int64_t l_sb, l_sn, l_sh;
    float* lse;
    int32_t* status;
    const int32_t* kv_len;         // optional per-batch key counts
    int B, Nq, Nk, H, Hkv;
    int causal;
    int shift;                     // key j is visible to query i iff j <= i + shift
    int n_pairs;                   // ceil(query tiles / 2)
    int items_per_head;            // causal: ceil(n_pairs / 2) mirrored items; else n_pairs
    int n_items;                   // items_per_head * B * H
    int wait_limit_ms;             // limit of one mbarrier wait (0: the default)
    float scale_log2;
    float scale;                   // PREC != 0: scores stay in natural units              // scale * log2(e)
    uint32_t drop_thr;
    float inv_keep;
    PhiloxKey key;
    DropoutOrigin rng;
    int d;                         // head size (PREC = 1: at most the template's D, a multiple of 8)
    const float* bias;             // PREC = 1: optional additive bias, element strides below (0 broadcasts)
    int64_t bias_sb, bias_sn, bias_sh;
    int bias_vec;                  // its rows can be read as float4
    int bias_b, bias_h;            // PREC = 2: whether it has a batch / head dimension
    const uint4* mq;               // DROP = 2: keep bits, [(b*H + h) * n_kblocks + key block][padded query row]
    int nq_pad, n_kblocks;
    // Rows of a query tile: `pack` query heads of one K/V head times `q_per_tile` queries, the heads fastest
    // (1 and 128 unless the call is packed, see plan_schedule()).  `heads` = H / pack columns per batch entry.
    int pack, q_per_tile, heads;
    // Split schedule: the call's (pair, key block) units are cut into gridDim.x equal ranges; a pair that lies in
    // several ranges leaves partial results for fwd_merge_kernel.
    int part_rows;                 // rows a partial's slot holds
    int start_cost;                // one tile: units a pair's start counts as, in front of its key blocks (plan_schedule)
    float4* part_o;                // [2 * gridDim.x slots][D / 4][part_rows], sums not yet divided
    float2* part_ml;               // [2 * gridDim.x slots][part_rows]: maximum (log2 units), row sum (< 0: no block visited)
    int4* part_meta;               // [gridDim.x]: batch, column, pair, number of ranges (0: none starts here)
};

// A stretch of work: key blocks [j0, j1) of a pair.  n[t]: blocks the pair's tile t has in all
// (0: no rows); count(t): how many of them lie in this stretch.
struct Stretch {
    int pair, h, b, nk, j0, j1, n[2];
    __device__ __forceinline__ int count(int t) const { const int e = n[t] < j1 ? n[t] : j1; return e > j0 ? e - j0 : 0; }
    __device__ __forceinline__ bool whole() const { return j0 == 0 && j1 >= n[0] && j1 >= n[1]; }
};

// key blocks tile t of a pair of tiles with q_per_tile queries visits
__device__ __forceinline__ int num_blocks(const FwdArgs& a, int q_per_tile, int pair, int t, int nk) {
    const int row0 = (pair * 2 + t) * q_per_tile;
    int kv_end = nk;               // keys this batch entry attends to
    if (a.causal && row0 + q_per_tile + a.shift < kv_end) kv_end = row0 + q_per_tile + a.shift;
    return (row0 < a.Nq) ? (kv_end + kBlockN - 1) / kBlockN : 0;
}
__device__ __forceinline__ int pair_blocks(const FwdArgs& a, int pair, int nk) {
    const int n0 = num_blocks(a, a.q_per_tile, pair, 0, nk), n1 = num_blocks(a, a.q_per_tile, pair, 1, nk);
    return n0 > n1 ? n0 : n1;
}

// Where a CTA's range of units starts and how long it is (split schedule), left in shared memory for every role.  A pair
// has start_cost units that stand for its start, then one for each key block; `at` is the range's place in its first pair.
// `ctas`: CTAs that have a range (with per-batch key counts the units can be fewer than the CTAs; every range has one).
struct RangeStart { int b, h, pair, at, units, total, ctas; };
__device__ __forceinline__ int range_begin(int cta, int ctas, int total) { return (int)((int64_t)cta * total / ctas); }

__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) { const int o = __shfl_up_sync(0xffffffffu, v, off); if (lane >= off) v += o; }
    return v;
}
// The index i < n whose cost range holds unit `target` of the costs laid end to end; target becomes the offset in it.
template <typename Cost>
__device__ __forceinline__ int warp_find(int n, int lane, int& target, Cost cost) {
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int c = i0 + lane < n ? cost(i0 + lane) : 0;
        const int incl = warp_scan(c, lane);
        const uint32_t hit = __ballot_sync(0xffffffffu, target < incl);
        if (hit) {
            const int l = __ffs((int)hit) - 1;
            target -= __shfl_sync(0xffffffffu, incl - c, l);
            return i0 + l;
        }
        target -= __shfl_sync(0xffffffffu, incl, 31);
    }
    return n - 1;
}
// The units of a pair that a walk with `units` left takes from place `at` on, as key blocks [j0, j1); returns what is left
// for the next pairs, nothing where it would end before a pair's first block (find_range sees to the first pair).
template <int SCHED> __device__ __forceinline__ int start_cost(const FwdArgs& a) { return SCHED == 2 ? a.start_cost : 0; }
template <int SCHED>
__device__ __forceinline__ int take_units(const FwdArgs& a, int at, int units, Stretch& s) {
    const int n = s.n[0] > s.n[1] ? s.n[0] : s.n[1], c0 = start_cost<SCHED>(a);
    s.j0 = max(at - c0, 0);
    s.j1 = min(n, at + units - c0);
    const int left = at + units - c0 - n;
    return left > c0 ? left : 0;
}
// One warp: the costs are the pairs' units; with per-batch key counts a batch entry has a total of its own.
template <int SCHED>
__device__ __forceinline__ void find_range(const FwdArgs& a, int lane, volatile RangeStart* out) {
    const int c0 = start_cost<SCHED>(a);
    auto column = [&](int b) {                       // units of one (batch, column): serial, every lane its own b
        const int nk = kv_len_of(a.kv_len, b, a.Nk);
        int sum = 0;
        for (int pr = 0; pr < a.n_pairs; ++pr) sum += pair_blocks(a, pr, nk) + c0;
        return sum;
    };
    int total = 0, col = 0;
    if (a.kv_len) {
        for (int b = lane; b < a.B; b += 32) total += a.heads * column(b);
        total = __shfl_sync(0xffffffffu, warp_scan(total, lane), 31);
    } else {
        for (int pr = lane; pr < a.n_pairs; pr += 32) col += pair_blocks(a, pr, a.Nk) + c0;
        col = __shfl_sync(0xffffffffu, warp_scan(col, lane), 31);
        total = a.B * a.heads * col;
    }
    const int ctas = total < (int)gridDim.x ? total : (int)gridDim.x;
    if ((int)blockIdx.x >= ctas) { if (lane == 0) out->units = 0; return; }
    const int first = range_begin((int)blockIdx.x, ctas, total);
    const int units = range_begin((int)blockIdx.x + 1, ctas, total) - first;
    int at = first, b;
    if (a.kv_len) {
        b = warp_find(a.B, lane, at, [&](int i) { return a.heads * column(i); });
        col = column(b);
    } else {
        b = at / (a.heads * col);
        at -= b * a.heads * col;
    }
    const int h = at / col;
    at -= h * col;
    const int nk = kv_len_of(a.kv_len, b, a.Nk);
    const int pair = warp_find(a.n_pairs, lane, at, [&](int i) { return pair_blocks(a, i, nk) + c0; });
    if (lane == 0) {
        out->b = b; out->h = h; out->pair = pair; out->at = at; out->units = at + units > c0 ? units : 0; out->total = total; out->ctas = ctas;
    }
}

// A role's walk over the CTA's work; every role runs one of its own and sees the same stretches:
//     for (WorkLoop<SCHED> wl(a, range); wl.more(a); wl.advance()) for (u = 0; u < wl.kSub; ++u) if (wl.get(a, u, st)) ...
// Two walks and not one with a switch, because the softmax threads have no register to spare: one walk for
// both made the kernel of whole pairs spill more and cost it 1-2 % (B4 N4096 H32 D128).
template <int SCHED> struct WorkLoop;
template <> struct WorkLoop<0> {       // whole pairs, round robin
    static constexpr int kSub = 2;     // causal: a pair and its mirror
    int w;
    __device__ __forceinline__ WorkLoop(const FwdArgs&, const volatile RangeStart*) : w(blockIdx.x) {}
    __device__ __forceinline__ bool more(const FwdArgs& a) const { return w < a.n_items; }
    __device__ __forceinline__ void advance() { w += gridDim.x; }
    __device__ __forceinline__ bool get(const FwdArgs& a, int u, Stretch& s) const {
        const int bh = w / a.items_per_head, slot = w - bh * a.items_per_head;
        int pair;
        if (a.causal) {
            const int heavy = a.n_pairs - 1 - slot;           // more key blocks: first
            if (u == 0) pair = heavy;
            else { if (slot == heavy) return false; pair = slot; }
        } else {
            if (u == 1) return false;
            pair = slot;
        }
        s.pair = pair;
        s.h = bh % a.H;
        s.b = bh / a.H;
        s.nk = kv_len_of(a.kv_len, s.b, a.Nk);
        s.n[0] = num_blocks(a, kBlockM, pair, 0, s.nk); s.n[1] = num_blocks(a, kBlockM, pair, 1, s.nk);
        s.j0 = 0;
        s.j1 = s.n[0] > s.n[1] ? s.n[0] : s.n[1];
        return true;
    }
};
template <int SCHED> struct WorkLoop {       // split schedule: the CTA's range of units
    static constexpr int kSub = 1;
    int b, h, pair, at, units;
    __device__ __forceinline__ WorkLoop(const FwdArgs&, const volatile RangeStart* r)
        : b(r->b), h(r->h), pair(r->pair), at(r->at), units(r->units) {}
    __device__ __forceinline__ bool more(const FwdArgs&) const { return units > 0; }
    __device__ __forceinline__ void advance() {}
    __device__ __forceinline__ bool get(const FwdArgs& a, int, Stretch& s) {
        s.pair = pair; s.h = h; s.b = b;
        s.nk = kv_len_of(a.kv_len, b, a.Nk);
        s.n[0] = num_blocks(a, a.q_per_tile, pair, 0, s.nk); s.n[1] = num_blocks(a, a.q_per_tile, pair, 1, s.nk);
        units = take_units<SCHED>(a, at, units, s);
        at = 0;
        if (++pair == a.n_pairs) { pair = 0; if (++h == a.heads) { h = 0; ++b; } }
        return true;
    }
};

// The softmax warps' form of the walk: its state and the current stretch lie in shared memory, a record per warp, and
// the epilogue reads the stretch again, so that no register holds them while a block's 128 scores are worked on.
// Held in registers, the D = 128 kernel spilled 424 bytes instead of 60 and the chunk below took 152 us instead of 112.
struct WalkRecord { int b, h, pair, at, units, cur_pair, cur_h, cur_b, cur_j0, cur_j1; };
template <int SCHED> struct SoftmaxLoop;
template <> struct SoftmaxLoop<0> : WorkLoop<0> {
    __device__ __forceinline__ SoftmaxLoop(const FwdArgs& a, const volatile RangeStart* r, volatile WalkRecord*) : WorkLoop<0>(a, r) {}
    __device__ __forceinline__ void again(const FwdArgs&, Stretch&) const {}
};
template <int SCHED> struct SoftmaxLoop {
    static constexpr int kSub = 1;
    volatile WalkRecord* rec;
    __device__ __forceinline__ SoftmaxLoop(const FwdArgs&, const volatile RangeStart* r, volatile WalkRecord* w) : rec(w) {
        rec->b = r->b; rec->h = r->h; rec->pair = r->pair; rec->at = r->at; rec->units = r->units;    // every lane the same
        __syncwarp();
    }
    __device__ __forceinline__ bool more(const FwdArgs&) const { return rec->units > 0; }
    __device__ __forceinline__ void advance() {}
    __device__ __forceinline__ bool get(const FwdArgs& a, int, Stretch& s) {
        int b = rec->b, h = rec->h, pair = rec->pair;
        const int at = rec->at, units = rec->units;
        s.pair = pair; s.h = h; s.b = b;
        s.nk = kv_len_of(a.kv_len, b, a.Nk);
        s.n[0] = num_blocks(a, a.q_per_tile, pair, 0, s.nk); s.n[1] = num_blocks(a, a.q_per_tile, pair, 1, s.nk);
        const int left = take_units<SCHED>(a, at, units, s);
        if (++pair == a.n_pairs) { pair = 0; if (++h == a.heads) { h = 0; ++b; } }
        __syncwarp();                                  // every lane has read
        rec->b = b; rec->h = h; rec->pair = pair; rec->at = 0; rec->units = left;
        rec->cur_pair = s.pair; rec->cur_h = s.h; rec->cur_b = s.b; rec->cur_j0 = s.j0; rec->cur_j1 = s.j1;
        __syncwarp();
        return true;
    }
    __device__ __forceinline__ void again(const FwdArgs& a, Stretch& s) const {
        s.pair = rec->cur_pair; s.h = rec->cur_h; s.b = rec->cur_b; s.j0 = rec->cur_j0; s.j1 = rec->cur_j1;
        s.nk = kv_len_of(a.kv_len, s.b, a.Nk);
        s.n[0] = num_blocks(a, a.q_per_tile, s.pair, 0, s.nk); s.n[1] = num_blocks(a, a.q_per_tile, s.pair, 1, s.nk);
    }
};

// P is stored as 2^(S c - m + kPShift): with the lazily refreshed maximum P <= 2^8, so the shifted value
// stays below 2^14 in fp16 and entries down to 2^-20 of the row's largest keep full precision.
constexpr float kPShift = 6.0f;
constexpr float kPScale = 64.0f;            // 2^kPShift

// log(x) rounded once: the hardware's base-2 logarithm is off by up to 2^-22 and would be the largest error of an lse.
__device__ __noinline__ float exact_log(float x) { return (float)log((double)x); }

// DROP: 0 no dropout; 1 the keep bits are drawn here, by the softmax threads (no workspace);
// 2 they are loaded from the workspace, where dropout_bits_kernel has written the call's bits.
// SCHED: see FwdCfg.
template <int D, bool BF16, int DROP, int PREC, int SCHED>
__global__ void __launch_bounds__(kThreads, 1)
fwd_sm100_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_bias, const FwdArgs a) {
    using Cfg = FwdCfg<D, PREC, SCHED>;
    constexpr bool FREE = SCHED != 0, TWIN = SCHED == 2;
    constexpr int ST = Cfg::kStages;
    constexpr int TILE = Cfg::kTileBytes;
    // tcgen05.mma kind::f16 wants A and B in one format (an fp16 A next to a bf16 B raises an
    // illegal-instruction fault).  P is always fp16; a bf16 V tile is converted to fp16 in shared memory.
    // With P as a pair (PREC = 1) P_hi + P_lo come in V's own format and nothing is converted.
    constexpr bool CONV = BF16 && PREC == 0;
    constexpr bool P_BF16 = BF16 && PREC != 0;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + Cfg::kQTiles * TILE;
    uint8_t* sV = sK + ST * TILE;
    uint8_t* sBias = sV + ST * TILE;            // PREC = 2
    uint64_t* bars = (uint64_t*)(sBias + Cfg::kBiasBytes);
    uint32_t* tmem_slot = (uint32_t*)(bars + Cfg::kNumBars);
    volatile uint32_t* abort_flag = (volatile uint32_t*)(tmem_slot + 1);
    [[maybe_unused]] float2* sMl = (float2*)((uint8_t*)(bars + Cfg::kNumBars) + 64);      // SCHED = 2: [128]
    volatile RangeStart* range = (volatile RangeStart*)(tmem_slot + 4);      // seven words of the 64 bytes behind the barriers

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0) {                        // a lane a barrier: one thread for all of them took a microsecond of the launch
        for (int i = lane; i < Cfg::kNumBars; i += 32) {
            const bool wg_bar = (i >= Cfg::kPFull && i < Cfg::kPFull + 2) || (i >= Cfg::kPHalf && i < Cfg::kPHalf + 2) ||
                                i == Cfg::kMlFull || i == Cfg::kORead || i >= Cfg::kBiasEmpty;
            const bool conv_bar = (i >= Cfg::kVConv && i < Cfg::kVConv + ST);
            mbar_init(&bars[i], wg_bar ? 4u : (conv_bar ? 2u : 1u));
        }
        if (lane == 0) wait_control_init(abort_flag, a.wait_limit_ms);
        fence_mbar_init();
        __syncwarp();
    }
    if (warp == 8) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == 9 && lane == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
    }
    if (FREE && warp == 11) find_range<SCHED>(a, lane, range);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (FREE) grid_launch_dependents();       // fwd_merge_kernel, which waits for this grid's end

    const int pack = FREE ? a.pack : 1, q_per_tile = FREE ? a.q_per_tile : kBlockM;
    if (warp >= 8) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
      if (warp == 9) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            int kvc = 0;                    // K/V blocks loaded so far (ring index = count % ST)
            int q_loads[2] = {0, 0};
            bool ok = true;
            const uint32_t q_bytes = FREE ? (uint32_t)(Cfg::kNBox * 128 * pack * q_per_tile) : TILE;
            for (WorkLoop<SCHED> wl(a, range); wl.more(a) && ok; wl.advance()) {
                for (int u = 0; u < wl.kSub && ok; ++u) {
                    Stretch st;
                    if (!wl.get(a, u, st)) continue;
                    const int hk = st.h * pack / (a.H / a.Hkv);
                    const int q0 = st.pair * 2 * q_per_tile;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (st.count(t) == 0) continue;
                        // Q_t of the previous pair must have been read by its last S MMA
                        ok = mbar_wait(&bars[Cfg::kQEmpty + t], ((uint32_t)q_loads[t] & 1u) ^ 1u, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(&bars[Cfg::kQFull + t], q_bytes);
#pragma unroll
                        for (int bx = 0; bx < Cfg::kNBox; ++bx)
                            tma_load_4d(sQ + t * TILE + bx * kBoxBytes, &map_q, &bars[Cfg::kQFull + t],
                                        bx * 64, st.h * pack, q0 + t * q_per_tile, st.b);
                        ++q_loads[t];
                    }
                    for (int j = st.j0; j < st.j1 && ok; ++j, ++kvc) {
                        const int s = kvc % ST;
                        const uint32_t ph = (uint32_t)(kvc / ST) & 1u;
                        ok = mbar_wait(&bars[Cfg::kKEmpty + s], ph ^ 1u, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(&bars[Cfg::kKFull + s], TILE);
#pragma unroll
                        for (int bx = 0; bx < Cfg::kNBox; ++bx)
                            tma_load_4d(sK + s * TILE + bx * kBoxBytes, &map_k, &bars[Cfg::kKFull + s],
                                        bx * 64, hk, j * kBlockN, st.b);
                        ok = mbar_wait(&bars[Cfg::kVEmpty + s], ph ^ 1u, abort_flag);
                        if (!ok) {
                            // K of this block is in flight: let it land before giving up shared memory
                            for (int spin = 0; spin < 4096 && !mbar_try_wait(&bars[Cfg::kKFull + s], ph); ++spin) {}
                            break;
                        }
                        mbar_expect_tx(&bars[Cfg::kVFull + s], TILE);
#pragma unroll
                        for (int bx = 0; bx < Cfg::kNBox; ++bx)
                            tma_load_4d(sV + s * TILE + bx * kBoxBytes, &map_v, &bars[Cfg::kVFull + s],
                                        bx * 64, hk, j * kBlockN, st.b);
                    }
                }
            }
            if (!ok) {
                // unwinding: let copies already issued land before the CTA gives up its
                // shared memory (bounded: a copy that has not landed by now never will)
                for (int s = 0; s < ST; ++s) {
                    const int nf = (kvc + ST - 1 - s) / ST;       // completed K+V fills of stage s
                    for (int spin = 0; spin < 4096 && nf > 0 &&
                         !mbar_try_wait(&bars[Cfg::kKFull + s], (uint32_t)(nf - 1) & 1u); ++spin) {}
                    for (int spin = 0; spin < 4096 && nf > 0 &&
                         !mbar_try_wait(&bars[Cfg::kVFull + s], (uint32_t)(nf - 1) & 1u); ++spin) {}
                }
                for (int t = 0; t < 2; ++t)
                    for (int spin = 0; spin < 4096 && q_loads[t] > 0 &&
                         !mbar_try_wait(&bars[Cfg::kQFull + t], (uint32_t)(q_loads[t] - 1) & 1u); ++spin) {}
            }
        }
        __syncwarp();
      } else if (warp == 8) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc_f16(BF16, BF16, kBlockM, kBlockN, false, false);
            // P, V: fp16, or as a pair the inputs' format and the head size in whole groups of 16 columns
            const uint32_t idesc_pv = PREC ? make_idesc_f16(P_BF16, P_BF16, kBlockM, (a.d + 15) & ~15, false, true)
                                           : make_idesc_f16(false, false, kBlockM, D, false, true);
            const uint32_t sQ_u = smem_u32(sQ), sK_u = smem_u32(sK), sV_u = smem_u32(sV);

            // Descriptors differ only in the 16-byte-granular start address held in their low
            // bits: build one per buffer here and add offsets in the issue loops, which keeps the
            // single issuing thread's instruction count per MMA small.
            const uint64_t dQ = make_smem_desc_sw128(sQ_u, 0, 1024);
            const uint64_t dK = make_smem_desc_sw128(sK_u, 0, 1024);
            const uint64_t dV = make_smem_desc_sw128(sV_u, kBoxBytes, 1024);
            auto issue_s = [&](int t, int ks) {
                const uint64_t a0 = dQ + (uint64_t)((t * TILE) >> 4), b0 = dK + (uint64_t)((ks * TILE) >> 4);
                const uint32_t d = tmem + (uint32_t)t * 128u;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const uint32_t off = ((uint32_t)(kk >> 2) * kBoxBytes + (uint32_t)(kk & 3) * 32u) >> 4;
                    if (PREC == 0 || kk * 16 < a.d) mma_ss_f16(d, a0 + off, b0 + off, idesc_s, kk > 0);
                }
            };
            // one 64-key half (hf = 0, 1) of O_t += P_t V_j
            auto issue_pv = [&](int t, int vs, bool acc, int hf) {
                const uint64_t b0 = dV + (uint64_t)((vs * TILE) >> 4);
                const uint32_t d = tmem + 256u + (uint32_t)t * 128u, a0 = tmem + (uint32_t)t * 128u;
#pragma unroll
                for (int k4 = 0; k4 < kBlockN / 32; ++k4) {
                    const int kk = hf * (kBlockN / 32) + k4;
                    const uint64_t b = b0 + (uint64_t)((kk * 2048) >> 4);
                    if constexpr (PREC == 0) {
                        mma_ts_f16(d, a0 + (uint32_t)kk * 8u, b, idesc_pv, (acc || kk > 0) ? 1u : 0u);
                    } else {
                        // a half's 64 score columns hold P_hi (32 columns of pairs) and P_lo (the other 32)
                        const uint32_t ah = a0 + (uint32_t)(hf * 64 + k4 * 8);
                        mma_ts_f16(d, ah, b, idesc_pv, (acc || kk > 0) ? 1u : 0u);
                        mma_ts_f16(d, ah + 32u, b, idesc_pv, 1u);
                    }
                }
            };

            int kvc = 0;                    // K/V blocks consumed so far
            int q_uses[2] = {0, 0};         // pairs that used tile t (Q_full phase)
            int p_waits[2] = {0, 0};        // P_t hand-offs so far (P_full phase)
            bool ok = true;
            for (WorkLoop<SCHED> wl(a, range); TWIN && wl.more(a) && ok; wl.advance()) {
                Stretch st;
                wl.get(a, 0, st);
                // one tile: block j of the stretch belongs to accumulator set j & 1
                const int nb = st.j1 - st.j0;
                ok = mbar_wait(&bars[Cfg::kQFull], (uint32_t)q_uses[0] & 1u, abort_flag);
                ++q_uses[0];
                auto s_block = [&](int j) {
                    const int c = kvc + j;
                    if (!mbar_wait(&bars[Cfg::kKFull + c % ST], (uint32_t)(c / ST) & 1u, abort_flag)) return false;
                    tc_fence_after_sync();
                    const uint64_t b0 = dK + (uint64_t)(((c % ST) * TILE) >> 4);
                    const uint32_t d = tmem + (uint32_t)(j & 1) * 128u;
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t off = ((uint32_t)(kk >> 2) * kBoxBytes + (uint32_t)(kk & 3) * 32u) >> 4;
                        mma_ss_f16(d, dQ + off, b0 + off, idesc_s, kk > 0);
                    }
                    mma_commit(&bars[Cfg::kSFull + (j & 1)]);
                    mma_commit(&bars[Cfg::kKEmpty + c % ST]);
                    if (j == nb - 1) mma_commit(&bars[Cfg::kQEmpty]);
                    return true;
                };
                if (ok) ok = s_block(0);
                if (ok && nb > 1) ok = s_block(1);
                for (int j = 0; j < nb && ok; ++j) {
                    const int t = j & 1, c = kvc + j, vs = c % ST;
                    ok = mbar_wait(&bars[(CONV ? Cfg::kVConv : Cfg::kVFull) + vs], (uint32_t)(c / ST) & 1u, abort_flag);
                    if (ok) ok = mbar_wait(&bars[Cfg::kPHalf + t], (uint32_t)p_waits[t] & 1u, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    issue_pv(t, vs, j > 1, 0);
                    ok = mbar_wait(&bars[Cfg::kPFull + t], (uint32_t)p_waits[t] & 1u, abort_flag);
                    if (!ok) break;
                    ++p_waits[t];
                    tc_fence_after_sync();
                    issue_pv(t, vs, j > 1, 1);
                    if (j + 2 >= nb) mma_commit(&bars[Cfg::kODone + t]);
                    mma_commit(&bars[Cfg::kVEmpty + vs]);
                    if (j + 2 < nb) ok = s_block(j + 2);
                }
                kvc += nb;
            }
            for (WorkLoop<SCHED> wl(a, range); !TWIN && wl.more(a) && ok; wl.advance()) {
                for (int u = 0; u < wl.kSub && ok; ++u) {
                    Stretch st;
                    if (!wl.get(a, u, st)) continue;
                    const int nblk[2] = {st.count(0), st.count(1)};
                    const int nmax = st.j1 - st.j0;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (nblk[t] == 0) continue;
                        if (ok) ok = mbar_wait(&bars[Cfg::kQFull + t], (uint32_t)q_uses[t] & 1u, abort_flag);
                        ++q_uses[t];
                    }
                    if (ok) ok = mbar_wait(&bars[Cfg::kKFull + kvc % ST], (uint32_t)(kvc / ST) & 1u, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (nblk[t] == 0) continue;
                        issue_s(t, kvc % ST);
                        mma_commit(&bars[Cfg::kSFull + t]);
                        if (nblk[t] == 1) mma_commit(&bars[Cfg::kQEmpty + t]);
                    }
                    mma_commit(&bars[Cfg::kKEmpty + kvc % ST]);

                    for (int j = 0; j < nmax && ok; ++j) {
                        const int vs = (kvc + j) % ST;
                        const uint32_t vph = (uint32_t)((kvc + j) / ST) & 1u;
                        const int ks = (kvc + j + 1) % ST;
                        const uint32_t kph = (uint32_t)((kvc + j + 1) / ST) & 1u;
                        bool k_ready = false;
                        ok = mbar_wait(&bars[(CONV ? Cfg::kVConv : Cfg::kVFull) + vs], vph, abort_flag);
                        if (!ok) break;
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            if (j < nblk[t]) {
                                // the first 64 keys of P_t arrive while the second 64 are still computed
                                ok = mbar_wait(&bars[Cfg::kPHalf + t], (uint32_t)p_waits[t] & 1u, abort_flag);
                                if (!ok) break;
                                tc_fence_after_sync();
                                issue_pv(t, vs, j > 0, 0);
                                ok = mbar_wait(&bars[Cfg::kPFull + t], (uint32_t)p_waits[t] & 1u, abort_flag);
                                if (!ok) break;
                                ++p_waits[t];
                                tc_fence_after_sync();
                                issue_pv(t, vs, j > 0, 1);
                                if (j == nblk[t] - 1) mma_commit(&bars[Cfg::kODone + t]);
                            }
                            if (t == 1) mma_commit(&bars[Cfg::kVEmpty + vs]);
                            if (j + 1 < nblk[t]) {
                                if (!k_ready) {
                                    ok = mbar_wait(&bars[Cfg::kKFull + ks], kph, abort_flag);
                                    if (!ok) break;
                                    k_ready = true;
                                    tc_fence_after_sync();
                                }
                                issue_s(t, ks);
                                mma_commit(&bars[Cfg::kSFull + t]);
                                if (j + 2 == nblk[t]) mma_commit(&bars[Cfg::kQEmpty + t]);   // last S of tile t
                            }
                        }
                        if (ok && j + 1 < nmax) mma_commit(&bars[Cfg::kKEmpty + ks]);
                    }
                    kvc += nmax;
                }
            }
        }
        __syncwarp();
      } else if (CONV) {
        // ------------------------------------------------------------ warps 10-11: V_j bf16 -> fp16
        // the same walk as the producer's; a tile is touched between its arrival (V_full) and its
        // first reader (the PV MMAs wait for V_conv instead of V_full)
        const int ct = (warp - 10) * 32 + lane;
        int kvc = 0;
        bool ok = true;
        for (WorkLoop<SCHED> wl(a, range); wl.more(a) && ok; wl.advance()) {
            for (int u = 0; u < wl.kSub && ok; ++u) {
                Stretch st;
                if (!wl.get(a, u, st)) continue;
                for (int j = st.j0; j < st.j1; ++j, ++kvc) {
                    const int sidx = kvc % ST;
                    ok = mbar_wait(&bars[Cfg::kVFull + sidx], (uint32_t)(kvc / ST) & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    convert_tile_bf16_to_f16<false>(sV + sidx * TILE, TILE, ct, 64, 1.f);
                    fence_proxy_async_smem();           // generic-proxy writes -> visible to the MMA's reads
                    mbar_arrive_warp(&bars[Cfg::kVConv + sidx]);
                }
            }
        }
      } else if constexpr (PREC == 2) {
        // ------------------------------------------------------------ warps 10-11: the bias chunks of tile 0, 1
        const int t = warp - 10;
        if (elect_one()) {
            constexpr int NB = Cfg::kBiasSlots;
            int slot = 0, done = 0;
            uint32_t ph = 1u;                   // the slots start empty
            bool ok = true;
            for (WorkLoop<SCHED> wl(a, range); wl.more(a) && ok; wl.advance()) {
                for (int u = 0; u < wl.kSub && ok; ++u) {
                    Stretch st;
                    if (!wl.get(a, u, st)) continue;
                    const int n = st.j0 + st.count(t), row = (st.pair * 2 + t) * kBlockM;
                    for (int c = st.j0 * 4; c < n * 4 && ok; ++c) {
                        ok = mbar_wait(&bars[Cfg::kBiasEmpty + t * NB + slot], ph, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(&bars[Cfg::kBiasFull + t * NB + slot], kBoxBytes);
                        tma_load_4d(sBias + (t * NB + slot) * kBoxBytes, &map_bias, &bars[Cfg::kBiasFull + t * NB + slot],
                                    c * 32, a.bias_h ? st.h : 0, row, a.bias_b ? st.b : 0);
                        ++done;
                        if (++slot == NB) { slot = 0; ph ^= 1u; }
                    }
                }
            }
            for (int s = 0; s < NB && !ok; ++s) {           // unwinding: the copies in flight land first
                const int nf = (done + NB - 1 - s) / NB;
                for (int spin = 0; spin < 4096 && nf > 0 &&
                     !mbar_try_wait(&bars[Cfg::kBiasFull + t * NB + s], (uint32_t)(nf - 1) & 1u); ++spin) {}
            }
        }
        __syncwarp();
      }   // fp16 inputs: warps 10-11 idle, they complete the third warpgroup
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
        // ------------------------------------------------------------ softmax + epilogue
        using T16 = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
        const int t = warp >> 2;
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + (uint32_t)t * 128u + lane_off;
        const uint32_t tO = tmem + 256u + (uint32_t)t * 128u + lane_off;
        static_assert(sizeof(WalkRecord) == 40, "kWalkBytes");
        volatile WalkRecord* walk = (volatile WalkRecord*)((uint8_t*)(bars + Cfg::kNumBars) + 64 + Cfg::kMlBytes) + warp;
        int s_waits = 0;                 // S_t hand-offs so far (S_full phase)
        int o_waits = 0;                 // pairs finished so far (O_done phase)
        [[maybe_unused]] int stretches = 0;
        [[maybe_unused]] int bias_slot = 0;       // PREC = 2: next chunk's slot and phase
        [[maybe_unused]] uint32_t bias_ph = 0u;
        bool ok = true;

        if (FREE && threadIdx.x == 0) a.part_meta[blockIdx.x] = make_int4(0, 0, 0, 0);
        for (SoftmaxLoop<SCHED> wl(a, range, walk); wl.more(a) && ok; wl.advance()) {
            for (int u = 0; u < wl.kSub && ok; ++u) {
                Stretch st;
                if (!wl.get(a, u, st)) continue;
                // blocks [j0, n) are mine, with one tile every other one of them
                constexpr int kStep = TWIN ? 2 : 1;
                const int tile = TWIN ? 0 : st.pair * 2 + t;
                const int first = st.j0 + (TWIN ? t : 0), n = TWIN ? st.j1 : st.j0 + st.count(t), nk = st.nk;
                // my row: query i of head h; a packed tile may hold rows of no query (row_ok() is false)
                int i = tile * q_per_tile + (FREE ? r / pack : r);
                int h = FREE ? st.h * pack + r % pack : st.h;
                auto row_ok = [&] { return i < a.Nq && (!FREE || r < pack * q_per_tile); };
                if (FREE && !st.whole()) {
                    // the slot my row's partial goes to: a range's first stretch takes slot 0 unless it starts a pair
                    const int64_t slot = 2 * (int64_t)blockIdx.x + (st.j0 == 0 ? 1 : 0);
                    if (!TWIN && n == st.j0 && row_ok()) a.part_ml[slot * a.part_rows + t * kBlockM + r] = make_float2(-INFINITY, -1.f);
                    if (threadIdx.x == 0 && st.j0 == 0) {
                        // the pair starts here and goes on in the ranges of the CTAs behind this one
                        const int total = range->total, ctas = range->ctas;
                        const int full = st.n[0] > st.n[1] ? st.n[0] : st.n[1];
                        const int end = range_begin((int)blockIdx.x + 1, ctas, total) + (full - st.j1);
                        int k = 1;
                        while (range_begin((int)blockIdx.x + k, ctas, total) < end) ++k;
                        a.part_meta[blockIdx.x] = make_int4(st.b, st.h, st.pair, k);
                    }
                }
                if (!TWIN && n == st.j0) continue;
                // a warp none of whose rows is a query of the call keeps the pipeline's hand-offs going and computes
                // nothing: its rows of P are whatever tensor memory holds, and no other row of O depends on them
                const bool idle = TWIN && __all_sync(0xffffffffu, !row_ok());
                const uint32_t bh = dropout_column(a.rng, st.b, h);
                float m = -INFINITY, l = 0.f;
                // my row of the bias (a row beyond Nq, whose results nobody keeps, reads the last one)
                const float* brow = nullptr;
                if (PREC == 1 && a.bias)
                    brow = a.bias + st.b * a.bias_sb + h * a.bias_sh + (int64_t)(i < a.Nq ? i : a.Nq - 1) * a.bias_sn;

                for (int j = first; j < n; j += kStep) {
                    // DROP = 2: the block's 128 keep bits of my row, asked for before the wait for S
                    uint4 kb4 = make_uint4(0u, 0u, 0u, 0u);
                    if constexpr (DROP == 2)
                        kb4 = a.mq[((int64_t)(st.b * a.H + h) * a.n_kblocks + j) * a.nq_pad + i];
                    ok = mbar_wait(&bars[Cfg::kSFull + t], (uint32_t)s_waits & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);      // the TMEM accesses below are warp-collective
                    if (!ok) break;
                    ++s_waits;
                    if (idle) {
                        mbar_arrive_warp(&bars[Cfg::kPHalf + t]);
                        mbar_arrive_warp(&bars[Cfg::kPFull + t]);
                        continue;
                    }
                    tc_fence_after_sync();
                    uint32_t sr[4][32];                    // the row's 128 scores, then its 128 probabilities
#define SF(c) __uint_as_float(sr[(c) >> 5][(c) & 31])
#define SSET(c, x) sr[(c) >> 5][(c) & 31] = __float_as_uint(x)
#pragma unroll
                    for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, sr[c]);
                    tmem_wait_ld();

                    const int col0 = j * kBlockN;
                    if constexpr (PREC != 0) {
                        // Scores in natural units, the bias added as it is and before the mask: masks of the type's lowest
                        // value, of -1e9 or of its largest have to keep x - m (and, in the backward, x - lse) what the
                        // subtraction gives, and bias * log2 e overflows or is rounded by more than a whole unit there.
#pragma unroll
                        for (int q4 = 0; q4 < 4; ++q4) {
                            if constexpr (PREC == 2) {
                                // my row of the chunk: 16-byte pieces, swizzled by the row (no bank conflicts)
                                const int at = t * Cfg::kBiasSlots + bias_slot;
                                ok = mbar_wait(&bars[Cfg::kBiasFull + at], bias_ph, abort_flag);
                                ok = __all_sync(0xffffffffu, ok);
                                if (!ok) break;
                                const uint8_t* chunk = sBias + at * kBoxBytes + r * 128;
#pragma unroll
                                for (int c = 0; c < 32; c += 4) {
                                    const float4 b4 = *reinterpret_cast<const float4*>(chunk + (((c >> 2) ^ (r & 7)) << 4));
                                    SSET(q4 * 32 + c, fmaf(SF(q4 * 32 + c), a.scale, b4.x));
                                    SSET(q4 * 32 + c + 1, fmaf(SF(q4 * 32 + c + 1), a.scale, b4.y));
                                    SSET(q4 * 32 + c + 2, fmaf(SF(q4 * 32 + c + 2), a.scale, b4.z));
                                    SSET(q4 * 32 + c + 3, fmaf(SF(q4 * 32 + c + 3), a.scale, b4.w));
                                }
                                mbar_arrive_read_done(&bars[Cfg::kBiasEmpty + at]);
                                if (++bias_slot == Cfg::kBiasSlots) { bias_slot = 0; bias_ph ^= 1u; }
                            } else if (a.bias) {
                                const float* bp = brow + col0 + q4 * 32;
                                if (a.bias_vec && col0 + q4 * 32 + 32 <= a.Nk) {
#pragma unroll
                                    for (int c = 0; c < 32; c += 4) {
                                        const float4 b4 = *reinterpret_cast<const float4*>(bp + c);
                                        SSET(q4 * 32 + c, fmaf(SF(q4 * 32 + c), a.scale, b4.x));
                                        SSET(q4 * 32 + c + 1, fmaf(SF(q4 * 32 + c + 1), a.scale, b4.y));
                                        SSET(q4 * 32 + c + 2, fmaf(SF(q4 * 32 + c + 2), a.scale, b4.z));
                                        SSET(q4 * 32 + c + 3, fmaf(SF(q4 * 32 + c + 3), a.scale, b4.w));
                                    }
                                } else {
#pragma unroll
                                    for (int c = 0; c < 32; ++c) {
                                        const float b1 = col0 + q4 * 32 + c < a.Nk ? bp[c] : 0.f;
                                        SSET(q4 * 32 + c, fmaf(SF(q4 * 32 + c), a.scale, b1));
                                    }
                                }
                            }
                        }
                    }
                    if (PREC == 2 && !ok) break;
                    const bool need_mask = (a.causal && col0 + kBlockN - 1 > tile * q_per_tile + a.shift) || (col0 + kBlockN > nk);
                    if (need_mask) {
                        // my row sees the block's first `seen` columns: keys below the count, at most i + shift
                        int seen = nk - col0;
                        if (a.causal && i + a.shift + 1 - col0 < seen) seen = i + a.shift + 1 - col0;
#pragma unroll
                        for (int c = 0; c < 128; ++c)
                            if (c >= seen) SSET(c, -INFINITY);
                    }
                    float mx0 = SF(0), mx1 = SF(1), mx2 = SF(2), mx3 = SF(3);
#pragma unroll
                    for (int c = 4; c < 128; c += 8) {          // 3-input max: one instruction per two scores
                        mx0 = max3(mx0, SF(c), SF(c + 1)); mx1 = max3(mx1, SF(c + 2), SF(c + 3));
                        if (c + 4 < 128) { mx2 = max3(mx2, SF(c + 4), SF(c + 5)); mx3 = max3(mx3, SF(c + 6), SF(c + 7)); }
                    }
                    // with a bias the scores are x already, without one x = S scale is left to the FMA that takes the maximum off
                    const float to_x = PREC == 0 ? a.scale_log2 : (PREC == 1 && !a.bias ? a.scale : 1.f);
                    const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * to_x;
                    const float m_new = fmaxf(m, mx);
                    const bool grow = (m_new - m) > (PREC ? kRescaleThreshold * kLn2 : kRescaleThreshold);   // first block: inf > 8
                    if (__any_sync(0xffffffffu, grow)) {
                        // 0 on the first block; a row may have seen nothing but -inf so far (a bias; a stretch of a pair)
                        const float alpha = ((PREC || FREE) && m_new == -INFINITY) ? 0.f : ex2(PREC ? (m - m_new) * kLog2e : m - m_new);
                        m = m_new;
                        l *= alpha;
                        if (j > first) {
                            // S_t(j) complete implies PV_t(j-1) complete (same issuing thread, in order)
#pragma unroll
                            for (int c0 = 0; c0 < D; c0 += 16) {        // (32 at a time: 512 bytes of spills)
                                uint32_t orr[16];
                                tmem_ld_32x16(tO + c0, orr);
                                tmem_wait_ld();
#pragma unroll
                                for (int c = 0; c < 16; ++c) orr[c] = __float_as_uint(__uint_as_float(orr[c]) * alpha);
                                tmem_st_32x16(tO + c0, orr);
                            }
                        }
                    }
                    uint64_t la = 0ull, lb = 0ull;             // {0.f, 0.f}
                    if constexpr (PREC != 0) {
                        // P = e^(x - m) as hi + lo (fp16: times 2^kPShift), base 2 and the shift behind the difference, which is
                        // small where P is not.  A row that has seen only -inf so far keeps m = -inf; 0 in its place lets its
                        // P come out as 0.
                        const float nm = m == -INFINITY ? 0.f : -m;
                        const uint64_t nm2 = f2_pack(nm, nm), log2e2 = f2_pack(kLog2e, kLog2e), up2 = f2_pack(kPScale, kPScale), to_x2 = f2_pack(to_x, to_x);
                        // (la, lb: four short chains, whose roundings lse shows)
#pragma unroll
                        for (int q4 = 0; q4 < 4; ++q4) {
                            if (q4 == 3) {
                                tmem_wait_st();                // the first half, stored a quarter ago
                                tc_fence_before_sync();
                                mbar_arrive_warp(&bars[Cfg::kPHalf + t]);
                            }
                            uint32_t hi[16], lo[16];
#pragma unroll
                            for (int cc = 0; cc < 32; cc += 2) {
                                const int c = q4 * 32 + cc;
                                float p0, p1;
                                f2_unpack(f2_mul(PREC == 1 ? f2_fma(f2_pack(SF(c), SF(c + 1)), to_x2, nm2) : f2_add(f2_pack(SF(c), SF(c + 1)), nm2), log2e2), p0, p1);
                                uint64_t p2 = f2_pack(ex2(p0), ex2(p1));
                                if (!P_BF16) p2 = f2_mul(p2, up2);
                                if (cc & 2) lb = f2_add(lb, p2); else la = f2_add(la, p2);
                                f2_unpack(p2, p0, p1);
                                if constexpr (DROP == 2) {
                                    const uint32_t word = q4 == 0 ? kb4.x : (q4 == 1 ? kb4.y : (q4 == 2 ? kb4.z : kb4.w));
                                    if (!((word >> cc) & 1u)) p0 = 0.f;
                                    if (!((word >> cc) & 2u)) p1 = 0.f;
                                } else if constexpr (DROP == 1) {
                                    if ((cc & 15) == 0)
                                        kb4.x = dropout_keep_bits(a.key, bh, (uint32_t)i, (uint32_t)(j * 8 + (c >> 4)), a.drop_thr);
                                    if (!((kb4.x >> (cc & 15)) & 1u)) p0 = 0.f;
                                    if (!((kb4.x >> (cc & 15)) & 2u)) p1 = 0.f;
                                }
                                pack2_pair<P_BF16>(p0, p1, hi[cc / 2], lo[cc / 2]);
                            }
                            tmem_st_32x16(tS + (q4 >> 1) * 64 + (q4 & 1) * 16, hi);
                            tmem_st_32x16(tS + (q4 >> 1) * 64 + 32 + (q4 & 1) * 16, lo);
                        }
                        float l0, l1;
                        f2_unpack(f2_add(la, lb), l0, l1);
                        l += l0 + l1;
                        tmem_wait_st();
                        tc_fence_before_sync();
                        mbar_arrive_warp(&bars[Cfg::kPFull + t]);
                        continue;
                    }
                    // P = 2^(S*c - m): packed FMAs; of every four probabilities two take the
                    // special-function unit and two either that unit or the polynomial on the FMA pipes.  Without
                    // dropout P is packed to 16 bits as it is produced and each 64-key half is
                    // stored to TMEM as soon as it is complete, so conversion and store latency
                    // overlap the exponentials of the other half.
                    const float ms = kPShift - (FREE && m == -INFINITY ? 0.f : m);     // nothing seen yet: P = 0
                    const uint64_t c2 = f2_pack(a.scale_log2, a.scale_log2), nm2 = f2_pack(ms, ms);
                    uint32_t pk[32];
#pragma unroll
                    for (int c = 0; c < 128; c += 4) {
                        if (DROP != 1 && c == 64) tmem_st_32x32(tS, pk);
                        if (DROP != 1 && c == 64 + kHalfSignalAt) {
                            // the first half's store has had these groups' time to complete
                            tmem_wait_st();
                            tc_fence_before_sync();
                            mbar_arrive_warp(&bars[Cfg::kPHalf + t]);
                        }
                        float x0, x1, x2, x3, p0, p1, p2, p3;
                        f2_unpack(f2_fma(f2_pack(SF(c), SF(c + 1)), c2, nm2), x0, x1);
                        f2_unpack(f2_fma(f2_pack(SF(c + 2), SF(c + 3)), c2, nm2), x2, x3);
                        p0 = ex2(x0); p1 = ex2(x1);
                        if ((c >> 2) % Cfg::kPolyPeriod == 0) ex2_poly2(x2, x3, p2, p3);
                        else { p2 = ex2(x2); p3 = ex2(x3); }
                        la = f2_add(la, f2_pack(p0, p1));
                        lb = f2_add(lb, f2_pack(p2, p3));
                        if constexpr (DROP == 1) {
                            SSET(c, p0); SSET(c + 1, p1); SSET(c + 2, p2); SSET(c + 3, p3);
                        } else {
                            if constexpr (DROP == 2) {
                                // dropped entries leave the MMA's operand, not the row sum above
                                const uint32_t word = (c >> 5) == 0 ? kb4.x : ((c >> 5) == 1 ? kb4.y : ((c >> 5) == 2 ? kb4.z : kb4.w));
                                const uint32_t kw = word >> (c & 31);
                                if (!(kw & 1u)) p0 = 0.f;
                                if (!(kw & 2u)) p1 = 0.f;
                                if (!(kw & 4u)) p2 = 0.f;
                                if (!(kw & 8u)) p3 = 0.f;
                            }
                            pk[(c & 63) / 2] = pack2<P_BF16>(p0, p1);
                            pk[(c & 63) / 2 + 1] = pack2<P_BF16>(p2, p3);
                        }
                    }
                    if constexpr (DROP != 1) tmem_st_32x32(tS + 32, pk);
                    {
                        float s0, s1, s2, s3;
                        f2_unpack(la, s0, s1); f2_unpack(lb, s2, s3);
                        l += (s0 + s1) + (s2 + s3);
                    }
                    if constexpr (DROP == 1) {
#pragma unroll
                        for (int g = 0; g < 8; ++g) {
                            const uint32_t bits = dropout_keep_bits(a.key, bh, (uint32_t)i, (uint32_t)(j * 8 + g), a.drop_thr);
#pragma unroll
                            for (int c = 0; c < 16; ++c)
                                if (!((bits >> c) & 1u)) SSET(g * 16 + c, 0.f);
                        }
#pragma unroll
                        for (int c0 = 0; c0 < 2; ++c0) {
                            uint32_t pk[32];
#pragma unroll
                            for (int c = 0; c < 32; ++c) pk[c] = pack2<P_BF16>(SF(c0 * 64 + 2 * c), SF(c0 * 64 + 2 * c + 1));
                            tmem_st_32x32(tS + c0 * 32, pk);
                        }
                    }
#undef SF
#undef SSET
                    tmem_wait_st();
                    tc_fence_before_sync();
                    if (DROP == 1) mbar_arrive_warp(&bars[Cfg::kPHalf + t]);
                    mbar_arrive_warp(&bars[Cfg::kPFull + t]);
                }
                if (!ok) break;

                // ---- epilogue: O_t / l -> 16 bit -> global, straight from registers
                if constexpr (FREE) {
                    wl.again(a, st);
                    i = (TWIN ? 0 : st.pair * 2 + t) * q_per_tile + r / pack;
                    h = st.h * pack + r % pack;
                }
                if (!TWIN || t == 0 || st.j1 - st.j0 > 1) {
                    ok = mbar_wait(&bars[Cfg::kODone + t], (uint32_t)o_waits & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    ++o_waits;
                    tc_fence_after_sync();
                }
                // one tile: O = w0 O_0 + w1 O_1, the other set's maximum and sum through shared memory.  The second
                // warpgroup goes on, and lets O_1 be overwritten, when the first has read both.
                [[maybe_unused]] float w0 = 1.f, w1 = 0.f;
                if constexpr (TWIN) {
                    const uint32_t ph = (uint32_t)stretches & 1u;
                    ++stretches;
                    if (t == 1) {
                        sMl[r] = make_float2(m, st.j1 - st.j0 > 1 ? l : -1.f);
                        tc_fence_before_sync();
                        mbar_arrive_warp(&bars[Cfg::kMlFull]);
                        ok = mbar_wait(&bars[Cfg::kORead], ph, abort_flag);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        continue;
                    }
                    ok = mbar_wait(&bars[Cfg::kMlFull], ph, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const float2 o1 = sMl[r];
                    if (o1.y >= 0.f || o1.y != o1.y) {          // (NaN: the row's result)
                        const float m01 = fmaxf(m, o1.x);
                        w0 = m == -INFINITY ? 0.f : ex2(m - m01);
                        w1 = o1.x == -INFINITY ? 0.f : ex2(o1.x - m01);
                        m = m01;
                        l = fmaf(l, w0, o1.y * w1);
                    }
                }
                // 32 columns of my row's sums
                auto load_o = [&](int c0, uint32_t (&orr)[32]) {
                    tmem_ld_32x32(tO + c0, orr);
                    if constexpr (TWIN) {
                        uint32_t o1[32];
                        tmem_ld_32x32(tO + 128u + c0, o1);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            const float x = __uint_as_float(orr[c]);
                            orr[c] = __float_as_uint(st.j1 - st.j0 > 1 ? fmaf(x, w0, __uint_as_float(o1[c]) * w1) : x);
                        }
                        if (c0 + 32 == D) {
                            tc_fence_before_sync();
                            mbar_arrive_warp(&bars[Cfg::kORead]);
                        }
                    } else {
                        tmem_wait_ld();
                    }
                };
                if (FREE && !st.whole()) {
                    // a part of the pair's keys: the sums as they are, four columns of neighbouring rows side by side
                    const int64_t slot = 2 * (int64_t)blockIdx.x + (st.j0 == 0 ? 1 : 0);
                    const int pr = t * kBlockM + r;
                    if (row_ok()) a.part_ml[slot * a.part_rows + pr] = make_float2(m, l);
                    float4* po = a.part_o + slot * (int64_t)(D / 4) * a.part_rows + pr;
#pragma unroll
                    for (int c0 = 0; c0 < D; c0 += 32) {
                        uint32_t orr[32];
                        load_o(c0, orr);
                        if (row_ok()) {
#pragma unroll
                            for (int g = 0; g < 8; ++g)
                                po[(int64_t)(c0 / 4 + g) * a.part_rows] =
                                    make_float4(__uint_as_float(orr[4 * g]), __uint_as_float(orr[4 * g + 1]),
                                                __uint_as_float(orr[4 * g + 2]), __uint_as_float(orr[4 * g + 3]));
                        }
                    }
                    continue;
                }
                const float inv = a.inv_keep / l;
                T16* orow = reinterpret_cast<T16*>(a.o) + (int64_t)st.b * a.o_sb + (int64_t)i * a.o_sn +
                            (int64_t)h * a.o_sh;
                T16* lrow = a.o_lo ? reinterpret_cast<T16*>(a.o_lo) + (int64_t)st.b * a.l_sb + (int64_t)i * a.l_sn +
                                         (int64_t)h * a.l_sh : nullptr;
#pragma unroll
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t orr[32];
                    load_o(c0, orr);
                    if (row_ok()) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            if (PREC != 0 && c0 + g * 8 >= a.d) break;
                            uint4 v4;
                            v4.x = pack2<BF16>(__uint_as_float(orr[g * 8 + 0]) * inv, __uint_as_float(orr[g * 8 + 1]) * inv);
                            v4.y = pack2<BF16>(__uint_as_float(orr[g * 8 + 2]) * inv, __uint_as_float(orr[g * 8 + 3]) * inv);
                            v4.z = pack2<BF16>(__uint_as_float(orr[g * 8 + 4]) * inv, __uint_as_float(orr[g * 8 + 5]) * inv);
                            v4.w = pack2<BF16>(__uint_as_float(orr[g * 8 + 6]) * inv, __uint_as_float(orr[g * 8 + 7]) * inv);
                            *reinterpret_cast<uint4*>(orow + c0 + g * 8) = v4;
                            if (lrow) {
                                // residual: the exact value minus what was just stored, rounded once more
                                const uint32_t hi[4] = {v4.x, v4.y, v4.z, v4.w};
                                uint32_t lo[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    float h0, h1;
                                    unpack2<BF16>(hi[e], h0, h1);
                                    lo[e] = pack2<BF16>(__uint_as_float(orr[g * 8 + 2 * e]) * inv - h0,
                                                        __uint_as_float(orr[g * 8 + 2 * e + 1]) * inv - h1);
                                }
                                *reinterpret_cast<uint4*>(lrow + c0 + g * 8) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                            }
                        }
                    }
                }
                if (row_ok()) a.lse[((int64_t)st.b * a.H + h) * a.Nq + i] = PREC ? m + exact_log(P_BF16 ? l : l * (1.f / kPScale))
                                                                                 : kLn2 * ((m - kPShift) + log2f(l));
                // the O_t reads above are complete (wait::ld); the next pair's first PV_t MMA waits for
                // this warpgroup's next P_t, so it cannot overwrite O_t earlier
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0 && *abort_flag) report_status(a.status, 1);
}

// Put together the pairs that the split schedule cut: block (c, y) takes 32 rows of the pair that starts in CTA c's
// range and goes on in others.  Its parts are read in the order of the ranges, so the result does not depend on
// which CTA finished first.  A lane holds one row, a warp every eighth group of eight columns.  What bounds it is the
// chain of its loads behind the end of the main kernel (whose CTAs leave no registers for it to wait in): a pair that was
// cut has two parts at least, and where those lie does not depend on which pair it is, so the first two parts' rows are
// under way together with the record that says so (one bf16 query for each of 32 sequences of up to 4096 keys, 32 heads on 8:
// 11.3 -> 9.4 us, the call 82.1 -> 79.7; 700 queries on 8892 keys: 15.4 -> 13.9, 108.7 -> 107.7).
template <int D, bool BF16>
__global__ void __launch_bounds__(256) fwd_merge_kernel(const FwdArgs a) {
    using T16 = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rr = (int)blockIdx.y * 32 + lane, t = rr / kBlockM, r = rr % kBlockM;
    if (r >= a.pack * a.q_per_tile) return;
    auto slot_of = [&](int k) { return 2 * ((int64_t)blockIdx.x + k) + (k == 0 ? 1 : 0); };
    constexpr int kGroups = (D / 8 + 7) / 8;           // column groups a warp takes
    constexpr int kAhead = 2;                          // parts read before the record (the last range's second: its first again)
    const int4 meta = a.part_meta[blockIdx.x];
    float2 ml_a[kAhead];
    float4 po_a[kAhead][kGroups][2];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
        const int64_t slot = slot_of((int)blockIdx.x + k < (int)gridDim.x ? k : 0);
        ml_a[k] = a.part_ml[slot * a.part_rows + rr];
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
#pragma unroll
            for (int y = 0; y < 2; ++y)
                po_a[k][g][y] = a.part_o[(slot * (int64_t)(D / 4) + (g * 8 + warp) * 2 + y) * a.part_rows + rr];
    }
    const int i = (meta.z * 2 + t) * a.q_per_tile + r / a.pack, h = meta.y * a.pack + r % a.pack, b = meta.x;
    if (meta.w == 0 || i >= a.Nq) return;
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) if (k < meta.w) m = fmaxf(m, ml_a[k].x);
#pragma unroll 8
    for (int k = kAhead; k < meta.w; ++k) m = fmaxf(m, a.part_ml[slot_of(k) * a.part_rows + rr].x);
    float acc[kGroups][8], l = 0.f;
#pragma unroll
    for (int g = 0; g < kGroups; ++g)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] = 0.f;
    auto add = [&](const float2 ml, auto&& part) {
        if (ml.y < 0.f) return;                        // none of the tile's blocks lay in this range
        const float w = ml.x == -INFINITY ? 0.f : ex2(ml.x - m);
        l = fmaf(w, ml.y, l);
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            const float4 x = part(g, 0), y = part(g, 1);
            acc[g][0] = fmaf(w, x.x, acc[g][0]); acc[g][1] = fmaf(w, x.y, acc[g][1]);
            acc[g][2] = fmaf(w, x.z, acc[g][2]); acc[g][3] = fmaf(w, x.w, acc[g][3]);
            acc[g][4] = fmaf(w, y.x, acc[g][4]); acc[g][5] = fmaf(w, y.y, acc[g][5]);
            acc[g][6] = fmaf(w, y.z, acc[g][6]); acc[g][7] = fmaf(w, y.w, acc[g][7]);
        }
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
        if (k < meta.w) add(ml_a[k], [&](int g, int y) { return po_a[k][g][y]; });
#pragma unroll 4
    for (int k = kAhead; k < meta.w; ++k) {
        const int64_t slot = slot_of(k);
        const float4* po = a.part_o + slot * (int64_t)(D / 4) * a.part_rows + rr;
        add(a.part_ml[slot * a.part_rows + rr], [&](int g, int y) { return po[(int64_t)((g * 8 + warp) * 2 + y) * a.part_rows]; });
    }
    const float inv = a.inv_keep / l;
    T16* orow = reinterpret_cast<T16*>(a.o) + (int64_t)b * a.o_sb + (int64_t)i * a.o_sn + (int64_t)h * a.o_sh;
    T16* lrow = a.o_lo ? reinterpret_cast<T16*>(a.o_lo) + (int64_t)b * a.l_sb + (int64_t)i * a.l_sn + (int64_t)h * a.l_sh : nullptr;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
        const int c0 = (g * 8 + warp) * 8;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float x0 = acc[g][2 * e] * inv, x1 = acc[g][2 * e + 1] * inv;
            float h0, h1;
            hi[e] = pack2<BF16>(x0, x1);
            unpack2<BF16>(hi[e], h0, h1);
            lo[e] = pack2<BF16>(x0 - h0, x1 - h1);
        }
        *reinterpret_cast<uint4*>(orow + c0) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (lrow) *reinterpret_cast<uint4*>(lrow + c0) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    if (warp == 0) a.lse[((int64_t)b * a.H + h) * a.Nq + i] = kLn2 * ((m - kPShift) + log2f(l));
}

// How a call's query rows are tiled and its work divided.
struct FwdPlan {
    int pack, q_per_tile, heads, n_pairs;
    int sched;                     // FwdCfg's SCHED
    int ctas, part_rows;           // split schedule: ranges, rows per slot
    int start_cost;                // FwdArgs
    size_t ml_off, meta_off, bytes;        // workspace: partial sums | maxima and row sums | ranges' pairs
};

// units (key blocks walked by a pair of tiles) of one (batch, column), every batch entry with Nk keys
int64_t column_units(const fa_b200_params& p, int q_per_tile, int n_pairs) {
    const int64_t nk_blocks = (p.Nk + kBlockN - 1) / kBlockN;
    if (!p.causal) return n_pairs * nk_blocks;
    int64_t sum = 0;
    for (int pr = 0; pr < n_pairs; ++pr) {
        const int64_t q_end = (int64_t)(2 * pr + 1) * q_per_tile < p.Nq ? (int64_t)(2 * pr + 2) * q_per_tile : (int64_t)(2 * pr + 1) * q_per_tile;
        const int64_t n = (q_end + p.causal_shift + kBlockN - 1) / kBlockN;
        sum += n < nk_blocks ? n : nk_blocks;
    }
    return sum;
}

// `free`: the caller gave scratch and leaves the division of the work to the library.
//
// Packing.  The query heads that share a K/V head read the same keys, so with few queries they belong into one tile:
// 128 / pack queries of `pack` = H / Hkv heads.  Taken when it leaves at least 5 % fewer (pair, key block) units;
// with many queries both forms have the same number and the plain one stays.
// Splitting.  Whole pairs dealt round robin leave SMs idle when there are few of them, or when one batch entry's many
// keys make its pairs long.  The call's units are then cut into one equal range per SM.  What that costs
// (partial sums through memory and a second launch) is about kMergeUnits units, so the ranges have to be that much
// shorter than the longest round-robin share, and a tenth.  B200, before -> after, both rules together:
// 32 requests of 2048-4096 keys, 1 query, H32 Hkv8 D128 bf16: 304 -> 80 us (403 MB of keys and values, 62 us at the
// copy rate); 1 request, 700 queries on 8892 keys, same heads: 240 -> 108 us (98 GFLOP, 60 us at cuBLAS's rate).
// Decoding as one pair per unit, without the one-tile kernel (SCHED = 2), took 116 us: S, softmax and P V of one tile
// are a serial chain of about 2.7 us a block, and two stages of K and V cover too little of the memory's latency.
// Key counts are on the device, so the rule sees Nk.  Ranges are as even for unequal counts as for equal ones, whole
// pairs are not, and a block of the one-tile kernel takes about three quarters of the other kernel's time: with counts
// its ranges are taken at that.  Whole pairs -> ranges, 148 requests, 1 query, H8 Hkv8 D128, Nk 4096 (eight whole pairs
// an SM): all counts 4096 516 -> 384 us, counts from half of it 418 -> 300, all 1024 119 -> 114, all 256 48 -> 61.
// Calls of several tiles have no such gain: 8 requests of 2048 queries on 2048 keys, H16 D128, all counts 2048
// 282 -> 292 us, from half of it 242 -> 283, so nothing is taken off there.
constexpr int kMergeUnits = 4;
// Starts.  Q, the first S and the epilogue of a pair take as long as three blocks of the one-tile kernel (4.5 of
// 1.3 us), and ranges equal in blocks alone are not equal in time where counts make some pairs short.  With counts a
// pair's start therefore counts as that many units there, unless ranges are so short (in blocks, by Nk) that hardly any
// holds a whole pair.  Ranges equal in blocks -> so, 1 query, counts from 1 to an eighth of the cache: 148 requests, H8
// Hkv8 D64, Nk 8192 109 -> 83 us, D128, Nk 4096 115 -> 101, 37 requests, H32 Hkv8 D128, Nk 4096 38 -> 30; 32 requests
// of 2048-4096 keys, H32 Hkv8 D128 84 -> 82.  Without counts pairs are alike, and in the kernel of several tiles the
// walk with starts took registers from the softmax (700 queries on 8892 keys 93 -> 100 us).
constexpr int kLongRange = 8;
FwdPlan plan_schedule(const fa_b200_params& p, int D, int sms, bool free) {
    FwdPlan pl;
    memset(&pl, 0, sizeof(pl));
    auto pairs_of = [&](int qpt) { return (int)(((int64_t)p.Nq + 2 * qpt - 1) / (2 * qpt)); };
    pl.pack = 1; pl.q_per_tile = kBlockM; pl.heads = p.H; pl.n_pairs = pairs_of(kBlockM);
    if (!free || sms <= 0 || p.Nq > (1 << 20) || dropout_threshold(p.dropout_p) != 0u) return pl;
    const int group = p.H / p.Hkv;
    int64_t col = column_units(p, kBlockM, pl.n_pairs);
    const int items = p.causal ? (pl.n_pairs + 1) / 2 : pl.n_pairs;              // per column: a pair, or a pair and its mirror
    const int64_t n_items = (int64_t)items * p.B * p.H;
    const int64_t whole = (n_items + sms - 1) / sms * ((col + items - 1) / items);
    if (group > 1 && group <= kBlockM) {
        const int qpt = kBlockM / group, pairs = pairs_of(qpt);
        const int64_t packed = column_units(p, qpt, pairs);
        if (packed * p.Hkv * 20 <= col * p.H * 19) { pl.pack = group; pl.q_per_tile = qpt; pl.heads = p.Hkv; pl.n_pairs = pairs; col = packed; }
    }
    const int64_t total = (int64_t)p.B * pl.heads * col;
    pl.ctas = (int)(total < sms ? total : sms);
    int64_t ranges = (total + pl.ctas - 1) / pl.ctas;
    const bool one_tile = p.Nq <= pl.q_per_tile;
    if (p.kv_lengths && one_tile) ranges = (3 * ranges + 3) / 4;
    if (total < (1 << 28) && whole * 9 > (ranges + kMergeUnits) * 10) {
        pl.sched = one_tile ? 2 : 1;
        pl.start_cost = p.kv_lengths && one_tile && ranges >= kLongRange ? 3 : 0;
        const int tiles = (int)(((int64_t)p.Nq + pl.q_per_tile - 1) / pl.q_per_tile);
        const int rows = tiles > 1 ? 2 * kBlockM : p.Nq * pl.pack;
        pl.part_rows = (int)align_up((size_t)rows, 32);
        const size_t slots = 2 * (size_t)pl.ctas * pl.part_rows;
        pl.ml_off = align_up(slots * D * sizeof(float), 256);
        pl.meta_off = pl.ml_off + align_up(slots * sizeof(float2), 256);
        pl.bytes = pl.meta_off + align_up((size_t)pl.ctas * sizeof(int4), 256);
        return pl;
    }
    return plan_schedule(p, D, sms, false);
}

template <int D, bool BF16, int PREC>
int launch(const fa_b200_params& p, void* ws, size_t ws_bytes) {
    const int d = p.D;
    const int sms = sm_count(p.device);
    if (sms <= 0) { set_error("cannot read the SM count of device %d", p.device); return FA_ECUDA; }
    FwdPlan plan = plan_schedule(p, D, sms, ws != nullptr);
    if (ws_bytes < plan.bytes || ((uintptr_t)ws & 255u) != 0) plan = plan_schedule(p, D, sms, false);
    const CUtensorMapDataType dt = BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap mq, mk, mv;
    int r;
    if ((r = cached_tmap_bnhd(&mq, p.q.ptr, dt, 2, p.B, p.Nq, p.H, d, p.q.stride_b, p.q.stride_n, p.q.stride_h, plan.q_per_tile, 64, true, plan.pack)) ||
        (r = cached_tmap_bnhd(&mk, p.k.ptr, dt, 2, p.B, p.Nk, p.Hkv, d, p.k.stride_b, p.k.stride_n, p.k.stride_h, 128, 64, true)) ||
        (r = cached_tmap_bnhd(&mv, p.v.ptr, dt, 2, p.B, p.Nk, p.Hkv, d, p.v.stride_b, p.v.stride_n, p.v.stride_h, 128, 64, true))) {
        set_error("cuTensorMapEncodeTiled failed (%d)", r);
        return FA_ECUDA;
    }
    CUtensorMap mb = mq;
    const int bias_b = p.bias.stride_b != 0 && p.B > 1, bias_h = p.bias.stride_h != 0 && p.H > 1;
    if (PREC == 2 && (r = cached_tmap_bnhd(&mb, p.bias.ptr, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, bias_b ? p.B : 1, p.Nq, bias_h ? p.H : 1, p.Nk,
                                           p.bias.stride_b, p.bias.stride_n, p.bias.stride_h, 128, 32, 1))) {
        set_error("cuTensorMapEncodeTiled failed for the bias (%d)", r);
        return FA_ECUDA;
    }
    FwdArgs a;
    a.bias_b = bias_b; a.bias_h = bias_h;
    a.o = p.o.ptr;
    a.o_sb = p.o.stride_b; a.o_sn = p.o.stride_n; a.o_sh = p.o.stride_h;
    a.o_lo = p.o_lo.ptr;
    a.l_sb = p.o_lo.stride_b; a.l_sn = p.o_lo.stride_n; a.l_sh = p.o_lo.stride_h;
    a.lse = p.lse;
    a.status = p.status_word;
    a.wait_limit_ms = p.wait_limit_ms;
    a.B = p.B; a.Nq = p.Nq; a.Nk = p.Nk; a.H = p.H; a.Hkv = p.Hkv;
    a.kv_len = p.kv_lengths;
    a.causal = p.causal;
    a.shift = p.causal ? p.causal_shift : 0;
    a.pack = plan.pack; a.q_per_tile = plan.q_per_tile; a.heads = plan.heads;
    a.n_pairs = plan.n_pairs;
    a.part_rows = plan.part_rows;
    a.start_cost = plan.start_cost;
    a.part_o = (float4*)ws;
    a.part_ml = (float2*)((char*)ws + plan.ml_off);
    a.part_meta = (int4*)((char*)ws + plan.meta_off);
    a.items_per_head = p.causal ? (a.n_pairs + 1) / 2 : a.n_pairs;
    const int64_t n_items = (int64_t)a.items_per_head * p.B * plan.heads;
    if (n_items > 0x7fffffff - 65536) { set_error("too many work items"); return FA_EUNSUPPORTED; }
    a.n_items = (int)n_items;
    a.scale_log2 = p.scale * kLog2e;
    a.scale = pair_score_scale(p);
    a.d = d;
    a.bias = (const float*)p.bias.ptr;
    a.bias_sb = p.bias.stride_b; a.bias_sn = p.bias.stride_n; a.bias_sh = p.bias.stride_h;
    a.bias_vec = (((uintptr_t)p.bias.ptr & 15u) == 0 && (p.bias.stride_b | p.bias.stride_n | p.bias.stride_h) % 4 == 0) ? 1 : 0;
    a.drop_thr = dropout_threshold(p.dropout_p);
    a.inv_keep = 1.f / (1.f - dropout_effective_p(p.dropout_p));
    a.key = philox_make_key(p.seed, p.offset);
    a.rng = dropout_origin_of(p);
    // dropout: with a bit buffer the call's keep bits are written there first (unless an earlier call
    // left them) and the kernel loads them
    int drop = a.drop_thr ? 1 : 0;
    a.mq = nullptr;
    a.nq_pad = (int)align_up((size_t)p.Nq, 128);
    a.n_kblocks = (int)(align_up((size_t)p.Nk, 128) / 128);
    const size_t bits_one = dropout_bits_bytes(p);
    if (drop && p.dropout_bits && p.dropout_bits_bytes >= bits_one) {
        if (!p.dropout_bits_ready) {
            void* by_key = p.dropout_bits_bytes >= 2 * bits_one ? (char*)p.dropout_bits + bits_one : nullptr;
            int rc = launch_dropout_bits(p, p.dropout_bits, by_key);
            if (rc) return rc;
        }
        a.mq = (const uint4*)p.dropout_bits;
        drop = 2;
    }
    auto kernel = drop == 2 ? fwd_sm100_kernel<D, BF16, 2, PREC, 0> : fwd_sm100_kernel<D, BF16, 0, PREC, 0>;
    if constexpr (PREC != 2) if (drop == 1) kernel = fwd_sm100_kernel<D, BF16, 1, PREC, 0>;      // bias_is_staged()
    int smem = FwdCfg<D, PREC, 0>::kSmemBytes;
    if constexpr (PREC == 0) {
        if (plan.sched == 1) kernel = fwd_sm100_kernel<D, BF16, 0, PREC, 1>;
        if (plan.sched == 2) { kernel = fwd_sm100_kernel<D, BF16, 0, PREC, 2>; smem = FwdCfg<D, PREC, 2>::kSmemBytes; }
    }
    {
        static std::mutex mu;
        static uint64_t done[5] = {0, 0, 0, 0, 0};
        FA_CUDA_CHECK(set_smem_limit_once(kernel, smem, p.device, &done[plan.sched ? 2 + plan.sched : drop], &mu));
    }
    const int grid = plan.sched ? plan.ctas : (a.n_items < sms ? a.n_items : sms);     // one persistent CTA per SM
    kernel<<<grid, kThreads, smem, (cudaStream_t)p.stream>>>(mq, mk, mv, mb, a);
    FA_CUDA_CHECK(cudaGetLastError());
    if constexpr (PREC == 0) if (plan.sched) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)plan.ctas, (unsigned)(plan.part_rows / 32));
        cfg.blockDim = dim3(256);
        cfg.stream = (cudaStream_t)p.stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fwd_merge_kernel<D, BF16>, a));
    }
    return FA_OK;
}


#ifndef FA_PAIR_INSTANCES
bool tensor_ok(const fa_b200_tensor& t, int64_t B, int64_t N, int64_t H) {
    if (((uintptr_t)t.ptr & 15u) != 0) return false;
    if (H > 1 && (t.stride_h % 8) != 0) return false;
    if (N > 1 && (t.stride_n % 8) != 0) return false;
    if (B > 1 && (t.stride_b % 8) != 0) return false;
    return true;
}

}  // namespace

// Which calls the tensor-core family covers.  `why` names the first reason it does not.
bool sm100_supports(const fa_b200_params& p, bool backward, const char** why) {
    if (p.dtype == FA_B200_F32) {
        // fp32: the forward has a tensor-core kernel (TF32 products taken three times); the backward has one that AUTO
        // takes when the caller offers scratch (sm100_f32_bwd_scratch_bytes), CUDA-core tiles otherwise
        if (backward) { *why = "the fp32 backward is served by the CUDA-core kernels"; return false; }
        return sm100_tf32_fwd_supports(p, why);
    }
    if (p.bias.ptr) { *why = "an additive bias is not served by the single-P kernels"; return false; }
    if (p.D != 64 && p.D != 128) { *why = "head_dim must be 64 or 128"; return false; }
    return sm100_pair_supports(p, backward, why);
}

// Which calls the pair instances (PREC = 1) cover: 16-bit inputs, any head size TMA can address rows of
// (16-byte pieces), with or without a bias.  The head sizes and bias calls were served by the CUDA-core
// tiles before: forward + backward of B4 N1024 H16 D96 causal bf16 took 5.82 ms there.
bool sm100_pair_supports(const fa_b200_params& p, bool backward, const char** why) {
    if (p.dtype != FA_B200_F16 && p.dtype != FA_B200_BF16) { *why = "dtype must be fp16 or bf16"; return false; }
    if (p.D % 8 != 0 || p.D > 128) { *why = "head_dim must be a multiple of 8, at most 128"; return false; }
    if (!(p.scale > 0.f) || !(p.scale < 1e30f)) { *why = "scale must be positive and finite"; return false; }
    if (p.B > 65535 || p.H > 65535) { *why = "batch and heads must be below 65536"; return false; }
    if (!tensor_ok(p.q, p.B, p.Nq, p.H) || !tensor_ok(p.k, p.B, p.Nk, p.Hkv) ||
        !tensor_ok(p.v, p.B, p.Nk, p.Hkv) || !tensor_ok(p.o, p.B, p.Nq, p.H) ||
        (p.o_lo.ptr && !tensor_ok(p.o_lo, p.B, p.Nq, p.H)) ||
        (backward && (!tensor_ok(p.d_o, p.B, p.Nq, p.H) || !tensor_ok(p.dq, p.B, p.Nq, p.H) ||
                      !tensor_ok(p.dk, p.B, p.Nk, p.Hkv) || !tensor_ok(p.dv, p.B, p.Nk, p.Hkv)))) {
        *why = "tensors must be 16-byte aligned with strides that are multiples of 8 elements";
        return false;
    }
    *why = "";
    return true;
}

int sm100_fwd(const fa_b200_params& p, void* ws, size_t ws_bytes) {
    if (p.dtype == FA_B200_F32) return sm100_tf32_fwd(p);
    if (p.dtype == FA_B200_BF16) return p.D == 128 ? launch<128, true, 0>(p, ws, ws_bytes) : launch<64, true, 0>(p, ws, ws_bytes);
    return p.D == 128 ? launch<128, false, 0>(p, ws, ws_bytes) : launch<64, false, 0>(p, ws, ws_bytes);
}
size_t sm100_fwd_workspace_bytes(const fa_b200_params& p) {
    return p.dtype == FA_B200_F32 ? 0 : plan_schedule(p, p.D, sm_count(p.device), true).bytes;
}
#else
}  // namespace

// Whether a call's bias comes to the kernels by TMA (PREC = 2): rows of whole 16-byte pieces, one per query.  Not where
// the kernels draw their dropout bits themselves (`bits`: the buffer they would load them from otherwise), whose masks
// take the room in shared memory.
bool bias_is_staged(const fa_b200_params& p, size_t bits) {
    if (!p.bias.ptr || p.bias.stride_n == 0 || ((uintptr_t)p.bias.ptr & 15u) != 0) return false;
    if ((p.bias.stride_b | p.bias.stride_n | p.bias.stride_h) % 4 != 0) return false;
    return dropout_threshold(p.dropout_p) == 0u || (p.dropout_bits && p.dropout_bits_bytes >= bits);
}

int sm100_pair_fwd(const fa_b200_params& p) {
    if (bias_is_staged(p, dropout_bits_bytes(p))) {
        if (p.dtype == FA_B200_BF16) return p.D > 64 ? launch<128, true, 2>(p, nullptr, 0) : launch<64, true, 2>(p, nullptr, 0);
        return p.D > 64 ? launch<128, false, 2>(p, nullptr, 0) : launch<64, false, 2>(p, nullptr, 0);
    }
    if (p.dtype == FA_B200_BF16) return p.D > 64 ? launch<128, true, 1>(p, nullptr, 0) : launch<64, true, 1>(p, nullptr, 0);
    return p.D > 64 ? launch<128, false, 1>(p, nullptr, 0) : launch<64, false, 1>(p, nullptr, 0);
}
#endif

}  // namespace fa
