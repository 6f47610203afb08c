// The 64-filter residual tower with the boards RESIDENT in shared memory (sm_100a).
//
// A 3x3 convolution never looks outside its own board (the padded row / column around every board is zero), and a
// board of up to 15x15 cells x 64 channels is 32 KB in bf16 or fp16.  So a CTA takes a board through ALL the layers
// without the activations leaving the SM: the epilogue threads write a layer's output in place, in the 128-byte-
// swizzled rows the next layer's MMA descriptors read (every MMA that reads a layer's input is complete when its
// accumulators are), and keep the residual of a block in TMEM.
//
// A GEMM row is a PAIR of neighbouring cells.  tcgen05.mma with N = 64 (one cell's output channels) takes 48 cycles
// for 128x64x16, 2/3 of the tensor cores' rate, N = 128 takes 64, the full rate.  So the even and the odd columns of a
// board lie in two planes (row y * HP + p holds cells x = 2p and x = 2p + 1), a tile is 128 pairs = one whole 15x15
// board, and the accumulator holds the odd cell's 64 channels beside the even cell's.  Of the four columns a pair of
// outputs sees, the outer two feed one output each (N = 64), the inner two feed both (N = 128, the weights of two
// neighbouring taps lie one after the other as they are):
//     O[p-1] x W(-1) -> even            E[p] x [W(-1) | W(0)] -> odd | even
//     E[p+1] x W(+1) -> odd             O[p] x [W(0) | W(+1)] -> odd | even
// 3 rows x 4 K steps x (48 + 64 + 64 + 48) = 2,688 cycles a board and layer instead of 3,456, every output still
// summed tap by tap in the order of the one-layer kernels, so the results are theirs bit for bit.
// Smaller boards share a tile (two 10x10, four 7x7 ones) when there are more boards than SMs.
//
//   * Two tiles are in flight per CTA, each with its own MMA-issuing warp: while one tile's accumulators are drained
//     and written back as the next layer's input, the tensor cores run the other (it runs two thirds of a layer
//     behind).  MMAs of one tile stay in one warp, so their order does not depend on the interleaving.
//   * Sixteen epilogue warps: a warp owns one TMEM lane quadrant, one parity and 32 of the 64 channels.
//   * Weights stream from L2 through a one-layer ring of three 24 KB blocks (three taps of one dy each): a block is
//     handed back by a tcgen05.commit of every issuer, and the loader refills it with the next layer's when all have
//     come in (it stands in for the issuer of an absent second tile).
//   * Tiles are assigned statically: CTA c takes tiles c, c + grid, c + 2 grid, ... two at a time, through three
//     buffers, so that a tile's output can leave by TMA while its successor's input comes in.
//   * The heads' 1x1 convolutions are one more layer (launch_head_conv gives the same bits): fp32 weights split into
//     three 16-bit terms, products exact, the largest term's in an accumulator of their own.
//   * Given Gomoku move histories instead of an input tensor, the epilogue threads write a board's input planes
//     straight into its buffer (a position's row is 17 ones or zeros): no encoder launch, no input tensor in HBM.
// There is no communication between CTAs, so this is an ordinary launch (and may be captured in a
// graph).  Every wait is bounded; a thread that gives up raises the device error word.
// What bounds it is shared memory: the operands of a pair of tiles and layer take 5,376 cycles of its 128 bytes a cycle,
// the rows written 512, the weights brought in 576 (biases read from there, as before, another 256: they are a kernel
// parameter now).  Measured (15x15, 21 layers): 6,500 cycles a layer for two tiles in flight (7,400 with a cell per
// GEMM row), 4,600 for a lone one (5,450).  From some hundred boards on the GPU runs at its 1,000 W limit (1.75 GHz in
// these kernels), which takes part of that back: 4,096 boards 1,290 -> 1,230 us cold, 1,390 -> 1,320 us sustained.
// 1 board 70 -> 58 us; the 32 / 32-channel heads' convolutions, 31-47 us as a launch of their own before, 2 us.
// With the issuing warp in its loop as a whole (a lone lane moves every MMA's descriptors to uniform registers), an
// evaluation on the device, 2 / 1-channel heads: 250 boards 99 -> 83 us, 1,024 boards 333 -> 280, 4,096 boards 1,218 ->
// 1,031 on a cool GPU, one board 65.6 -> 63.6.
#include "internal.h"
#include "sm100_ptx.cuh"
#include "head_conv.cuh"
#include <algorithm>
#include <cstring>

namespace ob200 {
namespace {

constexpr int kTileM = 128;
constexpr int kC = 64;
constexpr int kRowBytes = kC * 2;
constexpr int kTapBytes = kC * kRowBytes;            // 8,192: one tap of one layer
constexpr int kGuardRows = 16;                       // zero rows before / between / after the planes (>= HP + 1, a multiple of 8)
constexpr int kPlaneRows = kTileM + kGuardRows;
constexpr int kBufs = 3;
constexpr int kActBytes = (kGuardRows + 2 * kBufs * kPlaneRows) * kRowBytes;     // 112,640
constexpr int kTmemCols = 512;
constexpr int kSlotCols = 256;                       // per tile in flight: 128 accumulators, 64 residual, 64 more for the heads
constexpr int kResidualCol = 128;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (kEpiWarps + 3);       // warps 0-15: epilogue, 16-17: MMA issue, 18: weight loader
constexpr int kWGroups = 3;                          // the weight ring is handed over in groups of three taps
constexpr int kWGroupBytes = 3 * kTapBytes;          // 24,576
constexpr int kNumBars = 2 + 2 + 2 + 2 * kWGroups + 2 + 1;
constexpr int kMaxLayers = 27;                       // the biases of so many layers fit the kernel parameter
constexpr int kHeadMax = 64;                         // head channels that fit the extra layer
constexpr int kSmemBytes = kActBytes + 9 * kTapBytes + 2 * kHeadMax * 4 + kNumBars * 8 + 16 + 1024;
static_assert(kSmemBytes <= 232448, "the buffers do not fit shared memory");

// The biases of all layers, as a kernel parameter: constant memory, read by uniform loads.  Shared memory is what the
// kernel is short of (the MMAs' operands alone take 128 bytes a cycle), and every warp needs 32 biases a layer.
struct ResidentBias { float v[kMaxLayers * kC]; };

struct ResidentParams {
    const uint8_t* const* layers;   // [n_layers] packed weights (ob200_pack_conv3x3_weights): 9 taps x 8 KB
    int n_layers;
    int B, S, HP;
    int per_tile, tiles;      // boards per tile
    int board_rows;           // rows of a board in a plane: (S + 1) * HP
    int* error;
    // optional: the heads' 1x1 convolutions (+ folded BatchNorm, ReLU) on the tower's output.  head.hc == 0: none.
    HeadConvWeights head;
    int head_rows;            // head.hc rounded up to 16
    float *hp, *hv;           // [B][pitch]: channel c of a cell at c * S*S + cell
    int hp_pitch, hv_pitch;
    // optional: the tower's input comes from Gomoku move histories instead of an input tensor - the epilogue
    // threads write each board's input rows themselves (the planes of ob200_launch_encode_gomoku).  enc_hist == null: off.
    const int16_t* enc_hist;  // [B][16] k-th most recent move
    const uint8_t* enc_nh;    // [B]
    const uint8_t* enc_tm;    // [B] 1 BLACK, 2 WHITE
    int enc_planes;           // 17 or 19
};

using namespace ptx;

// The input row of one position from the board's move history, as encode_gomoku_board_kernel writes it
// (GomokuState::getEnhancedTensorRepresentation, reference src/games/gomoku/gomoku_state.cpp:223-262): plane p < 16
// is one where move k = p + 1 (p even) / p - 1 (p odd) of the history was played, plane 16 is one everywhere iff
// BLACK is to move, planes 17 / 18 (attack / defense) are zero as the reference's CPU code computes them.
// `half`: the 32 channels (four 16-byte chunks) this thread writes.
template <bool F16>
__device__ __forceinline__ void write_input_row(uint8_t* dst_row, int row, int half, int cell, const int16_t* hist, int nh, int tm, int planes) {
    uint32_t w[12] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};     // channels 0-23, two per word
    if (half == 0) {
        const uint4 ha = __ldg(reinterpret_cast<const uint4*>(hist)), hb = __ldg(reinterpret_cast<const uint4*>(hist) + 1);
        const uint32_t hw[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
        const uint32_t one = F16 ? 0x3C00u : 0x3F80u;
#pragma unroll
        for (int pl = 0; pl < 16; ++pl) {
            const int k = (pl & 1) ? pl - 1 : pl + 1;
            const int hk = (int)(int16_t)((k & 1) ? (hw[k >> 1] >> 16) : (hw[k >> 1] & 0xffffu));
            if (k < nh && hk == cell) w[pl >> 1] |= one << ((pl & 1) * 16);
        }
        if (planes > 16 && tm == 1) w[8] = one;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(dst_row + (((half * 4 + c) ^ (row & 7)) << 4)) =
            c < 3 ? make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]) : make_uint4(0u, 0u, 0u, 0u);
}

// PAIR: CTAs take their tiles two at a time (the general case).  When no CTA has more than one tile
// (batches up to the SM count) the barriers count one issuer only.
// F16: the boards and weights are fp16 instead of bf16 (same instruction, other operand-format bits).
template <bool PAIR, bool F16>
__global__ void __launch_bounds__(kThreads, 1)
conv_tower_resident_kernel(const __grid_constant__ CUtensorMap in_even, const __grid_constant__ CUtensorMap in_odd,
                           const __grid_constant__ CUtensorMap out_even, const __grid_constant__ CUtensorMap out_odd,
                           const __grid_constant__ ResidentBias bias, const ResidentParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* act_s = smem;                                 // [guard]([even plane][guard][odd plane][guard]) x 3
    uint8_t* w_s = act_s + kActBytes;                      // nine tap blocks of the current / next layer
    float* head_s = reinterpret_cast<float*>(w_s + 9 * kTapBytes);   // [64] scales, [64] biases
    uint64_t* bars = reinterpret_cast<uint64_t*>(head_s + 2 * kHeadMax);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar0 = smem_u32(bars);
    auto in_full = [&](int bd) { return bar0 + 8u * bd; };               // the tile's first input is in its buffer
    auto act_ready = [&](int bd) { return bar0 + 8u * (2 + bd); };       // the previous layer's output is written (or the heads' drained)
    auto acc_full = [&](int bd) { return bar0 + 8u * (4 + bd); };        // the tile's MMAs of this layer are complete
    auto w_full = [&](int g) { return bar0 + 8u * (6 + g); };
    auto w_empty = [&](int g) { return bar0 + 8u * (6 + kWGroups + g); };
    auto buf_free = [&](int bd) { return bar0 + 8u * (6 + 2 * kWGroups + bd); };       // the buffer the tile's successor goes to has been stored
    const uint32_t stagger = bar0 + 8u * (8 + 2 * kWGroups);             // tile 0 is far enough into the layer

    if (threadIdx.x == 0) {
        for (int bd = 0; bd < 2; ++bd) {
            mbar_init(in_full(bd), p.enc_hist ? kEpiWarps : 1); mbar_init(act_ready(bd), kEpiWarps); mbar_init(acc_full(bd), 1);
            mbar_init(buf_free(bd), 1);
        }
        // a weight block comes back from every issuer of a full round
        for (int g = 0; g < kWGroups; ++g) { mbar_init(w_full(g), 1); mbar_init(w_empty(g), PAIR ? 2 : 1); }
        mbar_init(stagger, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&in_even) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&in_odd) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&out_even) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&out_odd) : "memory");
    }
    // guards, pad rows and the rows of a plane beyond its boards are zero for the kernel's lifetime: nothing writes them
    // but the TMA loads, which bring zeros
    for (int i = threadIdx.x; i < kActBytes / 16; i += kThreads) reinterpret_cast<uint4*>(act_s)[i] = make_uint4(0u, 0u, 0u, 0u);
    if ((int)threadIdx.x < p.head.hc) {
        head_s[threadIdx.x] = p.head.scale[threadIdx.x];
        head_s[kHeadMax + threadIdx.x] = p.head.bias[threadIdx.x];
    }
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the zeros -> reads by the tensor cores / TMA
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    // this CTA's tiles: blockIdx.x, + gridDim.x, ...; two per round
    const int n_my = ((int)blockIdx.x < p.tiles) ? (p.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int rounds = (n_my + 1) / 2;
    const int L = p.n_layers;
    const bool heads = p.head.hc > 0;
    const int LL = L + (heads ? 1 : 0);
    auto tile_of = [&](int n) { return (int)blockIdx.x + n * (int)gridDim.x; };
    // byte offset of a plane of the n-th tile's buffer
    auto plane_off = [&](int n, int odd) { return (uint32_t)((kGuardRows + (2 * (n % kBufs) + odd) * kPlaneRows) * kRowBytes); };

    if (warp == kEpiWarps + 2) {
        // ---------------- weight loader ----------------
        // constants of the network: may start before the kernels ahead of this one in the stream are complete
        if (lane == 0) {
            bool ok = true;
            uint32_t uses[kWGroups] = {0u, 0u, 0u};
            for (int round = 0; ok && round < rounds; ++round) {
                // in a round with a single tile (the last one, when the CTA's tile count is odd) the loader stands in
                // for the issuer of the missing tile
                const bool alone = PAIR && (n_my & 1) && round == rounds - 1;
                for (int l = 0; ok && l < LL; ++l) {
                    const uint8_t* src = l < L ? p.layers[l] : p.head.w;
                    const uint32_t bytes = l < L ? (uint32_t)kWGroupBytes : (uint32_t)(3 * p.head_rows * kRowBytes);
#pragma unroll
                    for (int g = 0; g < kWGroups; ++g) {
                        if (l == L && g > 0) break;
                        if (alone && l > 0) mbar_arrive(w_empty(g));
                        if (uses[g] > 0 && !mbar_wait(w_empty(g), (uses[g] - 1) & 1u, abort_flag)) { ok = false; break; }
                        mbar_arrive_expect_tx(w_full(g), bytes);
                        bulk_g2s(smem_u32(w_s + g * kWGroupBytes), src + (size_t)g * kWGroupBytes, bytes, w_full(g));
                        ++uses[g];
                    }
                }
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.error, 4); }
        }
    } else if (warp >= kEpiWarps) {
        // ---------------- MMA issuers: warp 16 + bd for tile bd of the round ----------------
        // Tile 1 runs two thirds of a layer behind tile 0 (its issuer starts a layer when tile 0's has issued two of the
        // three weight blocks), so that one tile's MMAs cover the other's epilogue.
        // The warp runs the loop as a whole and one lane issues: with loop state the compiler knows to be the warp's, the
        // descriptors stay in uniform registers.
        const int bd = __shfl_sync(0xFFFFFFFFu, warp, 0) - kEpiWarps;
        if (PAIR || bd == 0) {
            const uint32_t lead = elect_one();
            constexpr uint32_t kIdesc64 = make_idesc(F16, kTileM, kC), kIdesc128 = make_idesc(F16, kTileM, 2 * kC);
            constexpr uint32_t kRow = kRowBytes >> 4, kTap = kTapBytes >> 4;
            const uint32_t w_lo = desc_lo(smem_u32(w_s));
            const uint32_t act_lo = desc_lo(smem_u32(act_s));
            const uint32_t d = tmem_base + (uint32_t)(bd * kSlotCols), d_odd = d, d_even = d + kC;
            const uint32_t dy_step = (uint32_t)p.HP * kRow;
            uint32_t ready_cnt = 0u, stagger_cnt = 0u, uses[kWGroups] = {0u, 0u, 0u};
            bool ok = true;
            for (int round = 0; ok && round < rounds; ++round) {
                const int n = 2 * round + bd;
                if (n >= n_my) break;                   // a single tile in the last round: tile 1's issuer is done
                const uint32_t even = act_lo + (plane_off(n, 0) >> 4), odd = act_lo + (plane_off(n, 1) >> 4);
                for (int l = 0; l < LL; ++l) {
                    if (l == 0 && !mbar_wait_warp(in_full(bd), (uint32_t)round & 1u, abort_flag)) { ok = false; break; }
                    if (round + l > 0) {
                        if (!mbar_wait_warp(act_ready(bd), ready_cnt & 1u, abort_flag)) { ok = false; break; }
                        ++ready_cnt;
                    }
                    if (l == L) {
                        // the heads' 1x1 convolutions: [W0 | W1] and, on top of W1's sums, W2
                        if (!mbar_wait_warp(w_full(0), uses[0] & 1u, abort_flag)) { ok = false; break; }
                        ++uses[0];
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const int hr = p.head_rows;
                        const uint32_t id2 = make_idesc(F16, kTileM, 2 * hr), id1 = make_idesc(F16, kTileM, hr);
#pragma unroll
                        for (int par = 0; par < 2; ++par)
#pragma unroll
                            for (int ks = 0; ks < kC / 16; ++ks) {
                                const uint32_t a = (par ? odd : even) + ks * 2, dh = d + (uint32_t)(par * 2 * hr);
                                umma_if(lead, dh, a, w_lo + ks * 2, id2, ks ? 1u : 0u);
                                umma_if(lead, dh + (uint32_t)hr, a, w_lo + (uint32_t)(2 * hr) * kRow + ks * 2, id1, 1u);
                            }
                        umma_commit_if(lead, w_empty(0));
                        umma_commit_if(lead, acc_full(bd));
                        continue;
                    }
                    if (bd == 1) {
                        if (!mbar_wait_warp(stagger, stagger_cnt & 1u, abort_flag)) { ok = false; break; }
                        ++stagger_cnt;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int dy = 0; dy < 3; ++dy) {
                        // weights are waited for and handed back three taps at a time (a wait costs the issuing
                        // thread about 50 cycles, a commit 25)
                        if (!mbar_wait_warp(w_full(dy), uses[dy] & 1u, abort_flag)) { ok = false; break; }
                        ++uses[dy];
                        const uint32_t e = even + (uint32_t)dy * dy_step - dy_step, o = odd + (uint32_t)dy * dy_step - dy_step;
                        const uint32_t w = w_lo + (uint32_t)(dy * 3) * kTap;
#pragma unroll
                        for (int ks = 0; ks < kC / 16; ++ks) umma_if(lead, d_even, o - kRow + ks * 2, w + ks * 2, kIdesc64, (dy | ks) ? 1u : 0u);
#pragma unroll
                        for (int ks = 0; ks < kC / 16; ++ks) {
                            if (dy == 0 && ks == 0) {          // the odd cells' sums start here, the even cells' have begun
                                umma_if(lead, d_odd, e, w, kIdesc64, 0u);
                                umma_if(lead, d_even, e, w + kTap, kIdesc64, 1u);
                            } else umma_if(lead, d, e + ks * 2, w + ks * 2, kIdesc128, 1u);
                        }
#pragma unroll
                        for (int ks = 0; ks < kC / 16; ++ks) umma_if(lead, d, o + ks * 2, w + kTap + ks * 2, kIdesc128, 1u);
#pragma unroll
                        for (int ks = 0; ks < kC / 16; ++ks) umma_if(lead, d_odd, e + kRow + ks * 2, w + 2 * kTap + ks * 2, kIdesc64, 1u);
                        umma_commit_if(lead, w_empty(dy));
                        if (PAIR && dy == 1 && bd == 0 && lead) mbar_arrive(stagger);
                    }
                    if (!ok) break;
                    umma_commit_if(lead, acc_full(bd));
                }
            }
            if (!ok && lead) { *abort_flag = 1; atomicExch(p.error, 2); }
        }
    } else {
        // ---------------- epilogue: TMEM -> registers -> the next layer's input rows, in place ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");   // inputs come from the kernels ahead in the stream
        const int q = warp & 3;                          // TMEM lane quadrant this warp may read
        const int half = (warp >> 2) & 1, par = warp >> 3;     // 32 of the 64 channels; 0 even, 1 odd cells
        const int row = q * 32 + lane;                   // row within the plane
        const int k_board = row / p.board_rows, r_in = row - k_board * p.board_rows;
        const int y = r_in / p.HP, x = 2 * (r_in - y * p.HP) + par;
        const bool on_board = k_board < p.per_tile && y < p.S && x < p.S;
        const int cell = y * p.S + x;
        const bool elected = threadIdx.x == 0;           // issues the tiles' loads and stores
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        const bool encode = p.enc_hist != nullptr;
        bool ok = true;
        // a tile's input: by TMA from the input tensor, or written here from its boards' move histories
        auto encode_tile = [&](int n) {
            const int board = tile_of(n) * p.per_tile + k_board;
            if (on_board && board < p.B)
                write_input_row<F16>(act_s + plane_off(n, par) + row * kRowBytes, row, half, cell, p.enc_hist + (size_t)board * 16,
                                     p.enc_nh[board], p.enc_tm[board], p.enc_planes);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // rows -> the tensor cores' reads
            __syncwarp();
            if (lane == 0) mbar_arrive(in_full(n & 1));
        };
        auto load_tile = [&](int n) {                    // elected thread
            const int board0 = tile_of(n) * p.per_tile, nb = min(p.per_tile, p.B - board0);
            mbar_arrive_expect_tx(in_full(n & 1), (uint32_t)(nb * 2 * p.board_rows * kRowBytes));
            for (int k = 0; k < nb; ++k) {
                const uint32_t at = smem_u32(act_s) + (uint32_t)(k * p.board_rows * kRowBytes);
                tma_load_4d(at + plane_off(n, 0), &in_even, 0, 0, 0, board0 + k, in_full(n & 1));
                tma_load_4d(at + plane_off(n, 1), &in_odd, 0, 0, 0, board0 + k, in_full(n & 1));
            }
        };
        auto store_tile = [&](int n) {                   // elected thread
            const int board0 = tile_of(n) * p.per_tile, nb = min(p.per_tile, p.B - board0);
            for (int k = 0; k < nb; ++k) {
                const uint32_t at = smem_u32(act_s) + (uint32_t)(k * p.board_rows * kRowBytes);
                tma_store_4d(&out_even, 0, 0, 0, board0 + k, at + plane_off(n, 0));
                tma_store_4d(&out_odd, 0, 0, 0, board0 + k, at + plane_off(n, 1));
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        };
        for (int n = 0; n < 2 && n < n_my; ++n) {
            if (encode) encode_tile(n);
            else if (elected) load_tile(n);
        }
        uint32_t full_cnt0 = 0u, full_cnt1 = 0u;          // acc_full phases seen; act_ready completes one phase for each
        for (int round = 0; ok && round < rounds; ++round) {
            const int nb = n_my - 2 * round >= 2 ? 2 : 1;
            for (int l = 0; ok && l < LL; ++l) {
                const bool even_layer = !(l & 1);
                const bool has_res = l >= 2 && even_layer && l < L, keep = even_layer && l + 2 < L;
                const float* bias_t = bias.v + (l * kC + __shfl_sync(0xffffffffu, half, 0) * 32);
                for (int bd = 0; bd < nb; ++bd) {
                    const int n = 2 * round + bd;
                    const uint32_t t_slot = tmem_base + lane_addr + (uint32_t)(bd * kSlotCols);
                    const uint32_t t_res = t_slot + (uint32_t)(kResidualCol + (par * 2 + half) * 16);
                    uint32_t res[16];
                    if (has_res) tmem_ld16(t_res, res);   // while the tile's MMAs still run
                    if (l < L) {                          // and the layer's biases come into the constant cache
#pragma unroll
                        for (int j = 0; j < 32; j += 8) asm volatile("" ::"f"(bias_t[j]));
                    }
                    const uint32_t phase = (bd ? full_cnt1 : full_cnt0) & 1u;
                    // every wait's outcome is voted on, so that a warp gives up as a whole (the TMEM loads below
                    // need all 32 lanes; the elected lane may come late from its store)
                    bool good = mbar_wait(acc_full(bd), phase, abort_flag);
                    if (!__all_sync(0xffffffffu, good)) { ok = false; break; }
                    if (bd) ++full_cnt1; else ++full_cnt0;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (l < L) {
                        uint8_t* dst_row = act_s + plane_off(n, par) + row * kRowBytes;
                        uint32_t r[32];
                        tmem_ld32(t_slot + (uint32_t)((par ? 0 : kC) + half * 32), r);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (has_res) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) asm volatile("" : "+r"(res[j]));   // no use of it may move above the wait
                        }
                        // relu(accumulator + bias [+ residual]); 16-byte chunk c of row r sits at chunk c ^ (r % 8)
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float4 b0 = *reinterpret_cast<const float4*>(bias_t + c * 8), b1 = *reinterpret_cast<const float4*>(bias_t + c * 8 + 4);
                            const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float v0 = __uint_as_float(r[c * 8 + 2 * j]) + bb[2 * j];
                                float v1 = __uint_as_float(r[c * 8 + 2 * j + 1]) + bb[2 * j + 1];
                                if (has_res) { float r0, r1; unpack2<F16>(res[c * 4 + j], r0, r1); v0 += r0; v1 += r1; }
                                res[c * 4 + j] = pack2_relu<F16>(v0, v1);
                            }
                            if (on_board)
                                *reinterpret_cast<uint4*>(dst_row + (((half * 4 + c) ^ (row & 7)) << 4)) =
                                    make_uint4(res[c * 4], res[c * 4 + 1], res[c * 4 + 2], res[c * 4 + 3]);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // rows -> the tensor cores' / the store's reads
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(act_ready(bd));
                        if (keep) {
                            tmem_st16(t_res, res);
                            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        }
                        if (l + 1 == L && elected) {
                            good = mbar_wait(act_ready(bd), phase, abort_flag);        // every warp has written its rows
                            if (good) store_tile(n);
                        }
                        if (l + 1 == L && !__all_sync(0xffffffffu, good)) { ok = false; break; }
                    } else {
                        // the heads' channels of this cell: eight at a time, alternating between the two halves
                        const int board = tile_of(n) * p.per_tile + k_board, S2 = p.S * p.S;
                        const bool real = on_board && board < p.B;
                        const uint32_t t_head = t_slot + (uint32_t)(par * 2 * p.head_rows);
                        for (int c = half; c < p.head_rows / 8; c += 2) {
                            uint32_t big[8], small[8];
                            tmem_ld8(t_head + c * 8, big);
                            tmem_ld8(t_head + p.head_rows + c * 8, small);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const int h = c * 8 + j;
                                if (h >= p.head.hc || !real) continue;
                                const float o = head_conv_value(__uint_as_float(big[j]), __uint_as_float(small[j]), head_s[h], head_s[kHeadMax + h]);
                                if (h < p.head.pc) p.hp[(size_t)board * p.hp_pitch + h * S2 + cell] = o;
                                else p.hv[(size_t)board * p.hv_pitch + (h - p.head.pc) * S2 + cell] = o;
                            }
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(act_ready(bd));
                    }
                    if (l + 1 == LL && n + 2 < n_my) {
                        // the successor's input goes into the buffer of tile n - 1: its MMAs are complete (its last accumulators
                        // have been waited for above), its store has read it when the elected thread says so
                        if (elected) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        if (!encode) { if (elected) load_tile(n + 2); }
                        else {
                            if (elected) mbar_arrive(buf_free(bd));
                            good = mbar_wait(buf_free(bd), (uint32_t)round & 1u, abort_flag);
                            if (!__all_sync(0xffffffffu, good)) { ok = false; break; }
                            encode_tile(n + 2);
                        }
                    }
                }
            }
        }
        if (elected) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // the output stores are complete
        if (!ok) { *abort_flag = 1; atomicExch(p.error, 3); }
    }

    // ---------------- teardown ----------------
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);    // copies in flight into shared memory land first
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
    }
}

}  // namespace

static int pairs_per_row(int S) { return (S + 2) / 2; }      // 2 HP >= S + 1: at least one zero column at the end of a row

// Whether a board of the size fits a tile, and the biases of so many layers their parameter.
bool tower_resident_covers(int S, int n_layers) {
    return S >= 1 && (S + 1) * pairs_per_row(S) <= kTileM && n_layers >= 1 && n_layers <= kMaxLayers;
}
int tower_resident_head_channels_max() { return kHeadMax; }

// The whole tower in one ordinary launch.  in / out: plane maps of the 64-channel input and output tensors;
// layers_dev: the layers' packed weights, n_layers pointers on the device; bias: [n_layers][64] on the host.
int launch_conv_tower_resident(const BoardPlaneMaps& in, const BoardPlaneMaps& out, const void* const* layers_dev, const float* bias, int n_layers, int B, int S,
                               cudaStream_t st, const HeadConvWeights* head, float* hp, float* hv, int hp_pitch, int hv_pitch,
                               int dtype, const int16_t* enc_hist, const uint8_t* enc_nh, const uint8_t* enc_tm, int enc_planes) {
    if (enc_hist && (!enc_nh || !enc_tm || (enc_planes != 17 && enc_planes != 19) || ((uintptr_t)enc_hist & 15)))
        return set_error(OB200_ERR_INVALID, "resident tower: bad move-history arguments (17 or 19 planes, histories 16-byte aligned)");
    if (!layers_dev || !bias || B <= 0) return set_error(OB200_ERR_INVALID, "resident tower: bad arguments");
    if (head && (head->hc < 1 || head->hc > kHeadMax || head->pc < 0 || head->pc > head->hc || !head->w || !head->scale || !head->bias ||
                 (head->pc > 0 && !hp) || (head->pc < head->hc && !hv)))
        return set_error(OB200_ERR_INVALID, "resident tower: bad head arguments");
    if (!tower_resident_covers(S, n_layers))
        return set_error(OB200_ERR_UNSUPPORTED, "resident tower: board size %d / %d layers do not fit", S, n_layers);
    if (int rc = require_device()) return rc;
    int dev = 0, sms = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    OB200_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    ResidentBias biases;
    std::memcpy(biases.v, bias, (size_t)n_layers * kC * sizeof(float));
    ResidentParams p{};
    p.layers = reinterpret_cast<const uint8_t* const*>(layers_dev); p.n_layers = n_layers; p.B = B; p.S = S; p.HP = pairs_per_row(S);
    p.board_rows = (S + 1) * p.HP;
    // small boards share a tile once there are more of them than SMs (the last board of a tile needs no pad row below it)
    p.per_tile = std::min((kTileM + p.HP) / p.board_rows, (B + sms - 1) / sms);
    p.tiles = (B + p.per_tile - 1) / p.per_tile;
    p.error = device_error_word();
    if (!p.error) return set_error(OB200_ERR_CUDA, "resident tower: cannot resolve the device error word");
    if (head) { p.head = *head; p.head_rows = (head->hc + 15) / 16 * 16; }
    p.hp = hp; p.hv = hv; p.hp_pitch = hp_pitch; p.hv_pitch = hv_pitch;
    p.enc_hist = enc_hist; p.enc_nh = enc_nh; p.enc_tm = enc_tm; p.enc_planes = enc_planes;
    const bool pair = p.tiles > sms;          // some CTA has two tiles or more
    const bool f16 = dtype == OB200_DTYPE_F16;
    auto kernel = f16 ? (pair ? conv_tower_resident_kernel<true, true> : conv_tower_resident_kernel<false, true>)
                      : (pair ? conv_tower_resident_kernel<true, false> : conv_tower_resident_kernel<false, false>);
    static bool configured[64][4] = {{false}};
    const int variant = f16 * 2 + pair;
    if (dev < 0 || dev >= 64 || !configured[dev][variant]) {
        OB200_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        if (dev >= 0 && dev < 64) configured[dev][variant] = true;
    }
    auto map = [](const BoardTensorMap& m) -> const CUtensorMap& { return *reinterpret_cast<const CUtensorMap*>(&m); };
    OB200_CUDA_OK(launch_dependent(kernel, dim3(std::min(p.tiles, sms)), dim3(kThreads), (size_t)kSmemBytes, st, map(in.even), map(in.odd),
                                   map(out.even), map(out.odd), biases, p));
    counters().launches.fetch_add(1, std::memory_order_relaxed);
    return OB200_OK;
}

}  // namespace ob200
