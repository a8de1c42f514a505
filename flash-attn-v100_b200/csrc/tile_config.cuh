// The one place the tensor-core kernels' tuned numbers live.  The kernels are compiled from these
// constants and fa_b200_tile_config() reports the same constants, so the table cannot disagree with
// the code.  Replaces the reference's run-time tuner and its per-bucket table
// (kernels/autotuning.py:289-474, config.py:288-348).  Every value is the best of an A/B on B200;
// the runs behind them are listed in the design notes.
#pragma once

namespace fa {
namespace tile {

constexpr int kBlockM = 128;            // query rows per tile
constexpr int kBlockN = 128;            // key rows per block

// ---- forward (fwd_sm100.cu) ---------------------------------------------------------------------
constexpr int kFwdQTilesPerCta = 2;     // two query tiles in flight: the softmax of one hides the MMAs of the other
constexpr int kFwdWarps = 12;           // 8 softmax + MMA + TMA + 2 converting (bf16) / spare (fp16) warps
constexpr int fwd_kv_stages(int D) { return D == 128 ? 2 : 4; }      // K and V rings: what 227 KB hold
constexpr int fwd_one_tile_kv_stages(int D) { return D == 128 ? 3 : 6; }   // one query tile: the other's room too
constexpr int fwd_bias_kv_stages(int D) { return D == 128 ? 1 : 2; }       // with a staged bias: its chunks take the room
constexpr int fwd_bias_slots(int D) { return D == 128 ? 3 : 4; }           // of 16 KB per query tile (a block has four)
constexpr int kFwdRegsSoftmax = 208;    // setmaxnreg split; best of 224/56, 216/72, 208/88, 200/104
constexpr int kFwdRegsOther = 88;
// One of fwd_poly_period(D) groups of four exponentials evaluates two by the polynomial on the FMA pipes instead of the
// special-function unit.  Cycles of a key block, both query tiles, N = 8192: D = 128 fp16 3030 without, 2960 with one of
// four, 2865 with one of two; D = 64 fp16 2960, 2717, 2905 (at half the MMAs a block the threads' instructions weigh more).
// The share also shows in the results' last bits, the polynomial being the less exact one: D = 64, one of four against one of
// two, error of lse against float64 0.60-0.88 of what it was (64 to 3001 tokens, both masks and types), o 0.998-1.000,
// gradients the same.
constexpr int fwd_poly_period(int D) { return D == 64 ? 4 : 2; }
constexpr int kFwdHalfSignalAt = 16;    // first half of P handed over after this many of the second half's exps
constexpr float kFwdRescaleLog2 = 8.f;  // the running maximum is refreshed when it grows by more than 2^8

// ---- backward (bwd_sm100.cu) --------------------------------------------------------------------
constexpr int kBwdWarpgroups = 4;       // elementwise warpgroups (2 -> 4: backward +11 %)
constexpr int kBwdWarps = 4 * kBwdWarpgroups + 4;                    // + MMA, TMA, warps 18 and 19 (bias and stores by TMA, conversions)
// ring depth of the streamed tiles: U is read by the first and the last MMA of its step (three
// stages took 16 % off the dQ kernel), W within one step; the key-stationary dropout instance at
// D = 128 gives 4 KB to its masks and keeps two and two
constexpr int bwd_u_stages(int D, bool masks) { return D == 64 ? 4 : (masks ? 2 : 3); }
constexpr int bwd_bias_u_stages(int D) { return D == 64 ? 4 : 2; }         // with a staged bias tile of 64 KB
constexpr int bwd_bias_w_stages(int D) { return D == 64 ? 3 : 1; }
constexpr int bwd_w_stages(int D) { return D == 64 ? 3 : 2; }
// the dQ kernel is launched programmatically behind the dK/dV kernel while one head's K and V take at
// most this many bytes (N = 4096 at D = 128: -1 % of the backward; longer sequences showed no gain)
constexpr long long kBwdOverlapMaxKvBytes = 4ll << 20;
// CTA order: (batch, head) columns per group such that a group's Q, K, V and dO fit this budget (half of L2)
constexpr long long kBwdGroupBytes = 64ll << 20;
// D = 64: one kernel for dK, dV and dQ (dQ tiles summed in global memory) unless the two-pass variant is asked for
constexpr bool bwd_one_kernel(int D) { return D == 64; }

}  // namespace tile
}  // namespace fa
