// 3x3 convolution of 128 / 256-channel towers on 8x8 boards (chess), as an implicit GEMM over real cells only.
//
// tower_wide.cu lays a GEMM over the padded 9 x 9 grid of a board, so that every tap is the same shared-memory tile read
// from another row: 81 rows for 64 cells, a fifth of the tensor cores' work spent on padding - and at large batches the
// chip runs at its power limit, where work is time.  Here a tile's rows are the cells themselves, ordered [y][board][x]:
//   * the taps' dy is a row shift by 8 * (boards of the unit), the rows above and below the board being zeros that TMA
//     fills in outside the map;
//   * the taps' dx is not a shift of the input at all: the three columns of a filter are three groups of 64 accumulator
//     columns (N = 192 = 3 dx x 64 output channels, K = 3 dy x C_in), and the epilogue adds the neighbours' sums,
//     out(x) = D-1(x - 1) + D0(x) + D+1(x + 1), by warp shuffles - the eight cells of a board row are eight lanes.
// An MMA of N = 192 reads 10 KB of shared memory in its 96 cycles (N = 128: 8 KB in 64, exactly the port's rate).
//
// A unit is 4 boards (two 128-row tiles: y 0-3 and 4-7) or, in small batches, 2 boards (one tile), times 64 output
// channels.  A 64-channel slice of the input is 10 TMA boxes (one per y, -1 ... 8); weights stream as 24 KB blocks
// ([dx][64 output channels] x 64 input channels of one dy) through a 4-deep ring.  Accumulators: one 256-column slot per
// tile in flight; two tiles run tile by tile in the first and the last slice, so that the drain of one tile hides under
// the MMAs of the other, and block by block in between, so that the ring is not held.
//
// Measured, a layer of 256 channels: 4,096 boards 235 -> 204 us, 64 boards 17.2 -> 8.9 us, one board 12.4 -> 8.0 us
// (the kernel over the padded grid with two tiles a CTA before).
// Large batches are bound by power and shared memory, small ones by the chain of 48 MMAs and the hand-over of a layer.
//
// Warp 0 loads activations, warp 2 weights, warp 1 issues the MMAs, warps 4-11 are two epilogue groups; tile q of a CTA
// goes to group and slot q % 2.  Every wait is bounded, as in tower_wide.cu.
#include "internal.h"
#include "sm100_ptx.cuh"
#include <algorithm>
#include <cstring>

namespace ob200 {
namespace {

constexpr int kS = 8, kTileM = 128, kNT = 64, kN = 3 * kNT;
constexpr int kSlice = 64, kRowBytes = kSlice * 2;
constexpr int kMaxBoards = 4;
constexpr int kAStageBytes = (kS + 2) * kMaxBoards * kS * kRowBytes;   // 40,960
constexpr int kAStages = 2;
constexpr int kBStageBytes = kN * kRowBytes;                            // 24,576
constexpr int kBStages = 4;
constexpr int kOutBytes = kTileM * kRowBytes;
constexpr int kGroups = 2;
constexpr int kSlotCols = 256, kTmemCols = kGroups * kSlotCols;
constexpr int kThreads = 128 + 128 * kGroups;
constexpr int kNumBars = 2 * kAStages + 2 * kBStages + 3 * kGroups;
constexpr int kSmemBytes = kAStages * kAStageBytes + kBStages * kBStageBytes + kGroups * kOutBytes + kNumBars * 8 + kNT * 4 + 16 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory of a CTA");

struct Board8Params {
    const uint8_t* w;         // packed weights: [part][k_slice][dy] blocks of 192 x 64
    const float* bias;
    int* error;
    int B, boards;            // boards of the batch, of a unit
    int part_shift;           // log2 of the parts of 64 output channels, each with its own CTAs
    int cta_units, more_units;   // a CTA of a part takes the next cta_units units, the first more_units CTAs one more
    int k_slices;
    int has_residual, relu;
};

using namespace ptx;
__device__ __forceinline__ void group_bar(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
// Barrier of an epilogue group that tells every thread whether any of them reports `bad`.
__device__ __forceinline__ bool group_any(int id, bool bad) {
    uint32_t r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 q, %2, 0;\nbar.red.or.pred p, %1, 128, q;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(r) : "r"(id), "r"((uint32_t)bad) : "memory");
    return r != 0;
}

template <bool F16>
__global__ void __launch_bounds__(kThreads, 1)
conv_board8_kernel(const __grid_constant__ CUtensorMap in_map, const __grid_constant__ CUtensorMap out_map,
                   const __grid_constant__ CUtensorMap res_map, const Board8Params p) {
    constexpr uint32_t kIdesc = make_idesc(F16, kTileM, kN);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* a_s = smem;
    uint8_t* b_s = a_s + kAStages * kAStageBytes;
    uint8_t* o_s = b_s + kBStages * kBStageBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(o_s + kGroups * kOutBytes);
    float* bias_s = reinterpret_cast<float*>(bars + kNumBars);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bias_s + kNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar0 = smem_u32(bars);
    auto afull_bar = [&](int s) { return bar0 + 8u * s; };
    auto aempty_bar = [&](int s) { return bar0 + 8u * (kAStages + s); };
    auto bfull_bar = [&](int s) { return bar0 + 8u * (2 * kAStages + s); };
    auto bempty_bar = [&](int s) { return bar0 + 8u * (2 * kAStages + kBStages + s); };
    auto accfull_bar = [&](int a) { return bar0 + 8u * (2 * kAStages + 2 * kBStages + a); };
    auto accempty_bar = [&](int a) { return bar0 + 8u * (2 * kAStages + 2 * kBStages + kGroups + a); };
    auto res_bar = [&](int g) { return bar0 + 8u * (2 * kAStages + 2 * kBStages + 2 * kGroups + g); };

    // (no division: the compiler must see that these are the same for all threads, as in tower_wide.cu)
    const int part = blockIdx.x & ((1 << p.part_shift) - 1), part_cta = blockIdx.x >> p.part_shift;
    const int unit0 = part_cta * p.cta_units + min(part_cta, p.more_units);
    const int unit1 = unit0 + p.cta_units + (part_cta < p.more_units ? 1 : 0);
    const int row_rows = p.boards * kS;          // rows of one y
    const int tiles = p.boards >> 1;              // tiles of a unit
    const int row_bytes = row_rows * kRowBytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kAStages; ++s) { mbar_init(afull_bar(s), 1); mbar_init(aempty_bar(s), 1); }
        for (int s = 0; s < kBStages; ++s) { mbar_init(bfull_bar(s), 1); mbar_init(bempty_bar(s), 1); }
        for (int a = 0; a < kGroups; ++a) { mbar_init(accfull_bar(a), 1); mbar_init(accempty_bar(a), 4); mbar_init(res_bar(a), 1); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&in_map) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&out_map) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&res_map) : "memory");
    }
    if (threadIdx.x < kNT) bias_s[threadIdx.x] = p.bias[part * kNT + threadIdx.x];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // Programmatic dependent launch: what reads or writes activations sits behind griddepcontrol.wait; the weight
    // ring fills while the previous layer drains.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == 0) {
        // ---------------- activation producer ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int it = 0;
            bool ok = true;
            for (int u = unit0; ok && u < unit1; ++u)
                for (int kc = 0; kc < p.k_slices; ++kc, ++it) {
                    const int s = it % kAStages;
                    if (!mbar_wait(aempty_bar(s), ((uint32_t)(it / kAStages) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_arrive_expect_tx(afull_bar(s), (uint32_t)((kS + 2) * row_bytes));
                    const uint32_t dst = smem_u32(a_s + s * kAStageBytes);
                    for (int y = 0; y < kS + 2; ++y)
                        tma_load_4d(dst + y * row_bytes, &in_map, kc * kSlice, 0, y - 1, u * p.boards, afull_bar(s));
                }
            if (!ok) { *abort_flag = 1; atomicExch(p.error, 1); }
        }
    } else if (warp == 2) {
        // ---------------- weight producer ----------------
        if (lane == 0) {
            const int blocks = p.k_slices * 3;
            const uint8_t* src = p.w + (size_t)part * blocks * kBStageBytes;
            int jt = 0;
            bool ok = true;
            for (int u = unit0; ok && u < unit1; ++u)
                for (int j = 0; j < blocks; ++j, ++jt) {
                    const int s = jt % kBStages;
                    if (!mbar_wait(bempty_bar(s), ((uint32_t)(jt / kBStages) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_arrive_expect_tx(bfull_bar(s), (uint32_t)kBStageBytes);
                    bulk_g2s(smem_u32(b_s + s * kBStageBytes), src + (size_t)j * kBStageBytes, (uint32_t)kBStageBytes, bfull_bar(s));
                }
            if (!ok) { *abort_flag = 1; atomicExch(p.error, 4); }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        {
            const uint32_t lead = elect_one();
            const uint32_t a_base = desc_lo(smem_u32(a_s)), b_base = desc_lo(smem_u32(b_s));
            const uint32_t dy_step = (uint32_t)row_bytes >> 4;
            constexpr uint32_t kTileStep = kOutBytes >> 4;
            int sa = 0, jt = 0, q = 0;
            uint32_t pha = 0;
            bool ok = true;
            auto b_at = [&](int j) { return b_base + (uint32_t)(j % kBStages) * (kBStageBytes >> 4); };
            auto b_wait = [&](int j) {
                const bool r = mbar_wait_warp(bfull_bar(j % kBStages), (uint32_t)(j / kBStages) & 1u, abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return r;
            };
            for (int u = unit0; ok && u < unit1; ++u, q += tiles) {
                for (int kc = 0; ok && kc < p.k_slices; ++kc, jt += 3) {
                    const bool first = kc == 0, last = kc == p.k_slices - 1;
                    if (!mbar_wait_warp(afull_bar(sa), pha, abort_flag)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_lo = a_base + (uint32_t)(sa * (kAStageBytes >> 4));
                    if (tiles == 2 && !first && !last) {
#pragma unroll
                        for (int dy = 0; dy < 3; ++dy) {
                            if (!b_wait(jt + dy)) { ok = false; break; }
                            const uint32_t b_lo = b_at(jt + dy), at = a_lo + dy * dy_step;
#pragma unroll
                            for (int t = 0; t < 2; ++t)
#pragma unroll
                                for (int ks = 0; ks < kSlice / 16; ++ks)
                                    umma_if(lead, tmem_base + (uint32_t)(t * kSlotCols), at + (uint32_t)(t * kTileStep + ks * 2), b_lo + (uint32_t)(ks * 2), kIdesc, 1u);
                            umma_commit_if(lead, bempty_bar((jt + dy) % kBStages));
                        }
                    } else {
                        for (int t = 0; ok && t < tiles; ++t) {
                            const int slot = (q + t) & 1;
                            const uint32_t d = tmem_base + (uint32_t)(slot * kSlotCols);
                            if (first) {
                                if (!mbar_wait_warp(accempty_bar(slot), ((uint32_t)((q + t) >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            }
#pragma unroll
                            for (int dy = 0; dy < 3; ++dy) {
                                if (t == 0 && !b_wait(jt + dy)) { ok = false; break; }
                                const uint32_t b_lo = b_at(jt + dy), at = a_lo + dy * dy_step + (uint32_t)t * kTileStep;
#pragma unroll
                                for (int ks = 0; ks < kSlice / 16; ++ks)
                                    umma_if(lead, d, at + (uint32_t)(ks * 2), b_lo + (uint32_t)(ks * 2), kIdesc, (dy | ks) ? 1u : (uint32_t)!first);
                                if (t == tiles - 1) umma_commit_if(lead, bempty_bar((jt + dy) % kBStages));
                            }
                            if (ok && last) umma_commit_if(lead, accfull_bar(slot));
                        }
                    }
                    if (ok) umma_commit_if(lead, aempty_bar(sa));
                    if (++sa == kAStages) { sa = 0; pha ^= 1u; }
                }
            }
            if (!ok && lead) { *abort_flag = 1; atomicExch(p.error, 2); }
        }
    } else if (warp >= 4) {
        // ---------------- epilogue ----------------
        const int group = (warp - 4) >> 2, quad = warp & 3;
        const int row = quad * 32 + lane, x = lane & 7;
        const bool leader = ((warp - 4) & 3) == 0 && lane == 0;
        const bool has_res = p.has_residual != 0;
        const int ys = kTileM / row_rows;                  // board rows of a tile
        const int board_of_row = row % row_rows / kS;
        uint8_t* stage_out = o_s + group * kOutBytes;
        const uint32_t stage_u32 = smem_u32(stage_out);
        uint32_t res_phase = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int total = (unit1 - unit0) * tiles;
        for (int q = group; q < total; q += kGroups) {
            const int u = unit0 + q / tiles, y0 = q % tiles * ys, board0 = u * p.boards;
            const bool valid = board0 + board_of_row < p.B;
            if (leader) {
                // the previous store of this group must have finished reading the staging tile
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                if (has_res) {
                    mbar_arrive_expect_tx(res_bar(group), (uint32_t)kOutBytes);
                    for (int y = 0; y < ys; ++y)
                        tma_load_4d(stage_u32 + y * row_bytes, &res_map, part * kNT, 0, y0 + y, board0, res_bar(group));
                }
            }
            if (group_any(1 + 2 * group, !mbar_wait(accfull_bar(group), (uint32_t)(q >> 1) & 1u, abort_flag))) {
                *abort_flag = 1; atomicExch(p.error, 3); break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (has_res) {
                if (group_any(1 + 2 * group, !mbar_wait(res_bar(group), res_phase, abort_flag))) { *abort_flag = 1; atomicExch(p.error, 5); break; }
                res_phase ^= 1u;
            }
            const uint32_t t_acc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(group * kSlotCols);
            uint8_t* my_row = stage_out + row * kRowBytes;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t m[32], c[32], n[32];              // the sums of the filter's left, middle and right column
                tmem_ld32(t_acc + (uint32_t)(h * 32), m);
                tmem_ld32(t_acc + (uint32_t)(kNT + h * 32), c);
                tmem_ld32(t_acc + (uint32_t)(2 * kNT + h * 32), n);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (h == 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty_bar(group));
                }
                const float* bias_t = bias_s + h * 32;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    // 128-byte swizzle of the staging tile: 16-byte chunk k of row r sits at chunk k ^ (r % 8)
                    uint4* slot = reinterpret_cast<uint4*>(my_row + (((h * 4 + k) ^ (row & 7)) << 4));
                    const uint4 rv = has_res ? *slot : make_uint4(0u, 0u, 0u, 0u);
                    const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
                    uint32_t ow[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float v[2], r[2];
                        unpack2<F16>(rw[j], r[0], r[1]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int i = k * 8 + j * 2 + e;
                            const float left = __uint_as_float(__shfl_up_sync(0xFFFFFFFFu, m[i], 1));
                            const float right = __uint_as_float(__shfl_down_sync(0xFFFFFFFFu, n[i], 1));
                            float s = __uint_as_float(c[i]);
                            if (x > 0) s += left;
                            if (x < kS - 1) s += right;
                            v[e] = s + bias_t[i] + r[e];
                            if (p.relu) v[e] = fmaxf(v[e], 0.0f);
                        }
                        ow[j] = pack2<F16>(v[0], v[1]);
                        if (!valid) ow[j] = 0u;
                    }
                    *slot = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            group_bar(2 + 2 * group);
            if (leader) {
                for (int y = 0; y < ys; ++y)
                    tma_store_4d(&out_map, part * kNT, 0, y0 + y, board0, stage_u32 + y * row_bytes);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    // ---------------- teardown ----------------
    if (*abort_flag) {
        // give copies that may still be in flight time to land before the shared memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
}

}  // namespace

bool conv_board8_covers(int S, int cin, int cout) { return S == kS && conv_wide_covers(cin, cout); }

int launch_conv_board8(const BoardRowMaps& in, const BoardRowMaps& out, const BoardRowMaps* res, const void* packed_w, const float* bias,
                       int B, int cin, int cout, int relu, cudaStream_t st, int dtype) {
    if (!packed_w || !bias || B <= 0) return set_error(OB200_ERR_INVALID, "conv (8x8): null pointer or empty batch");
    if (!conv_wide_covers(cin, cout)) return set_error(OB200_ERR_UNSUPPORTED, "conv (8x8): %d -> %d channels is not covered", cin, cout);
    if (int rc = require_device()) return rc;
    static bool configured[64] = {false};
    int dev = 0, sms = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        OB200_CUDA_OK(cudaFuncSetAttribute(conv_board8_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        OB200_CUDA_OK(cudaFuncSetAttribute(conv_board8_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    OB200_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    Board8Params p;
    p.w = static_cast<const uint8_t*>(packed_w); p.bias = bias; p.B = B;
    p.error = device_error_word();
    if (!p.error) return set_error(OB200_ERR_CUDA, "conv (8x8): cannot resolve the device error word");
    const int parts = cout / kNT;
    p.part_shift = parts == 4 ? 2 : 1; p.k_slices = cin / kSlice; p.has_residual = res != nullptr; p.relu = relu;
    // two boards a unit while that leaves no CTA with a second one (half the time of a unit of four); beyond, a weight
    // block that two tiles share is worth more
    const int ctas = std::max(1, sms / parts);
    p.boards = (B + 1) / 2 <= ctas ? 2 : 4;
    const int units = (B + p.boards - 1) / p.boards, part_ctas = std::min(units, ctas);
    p.cta_units = units / part_ctas; p.more_units = units % part_ctas;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts * part_ctas); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = kSmemBytes; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const int i = p.boards == 4;
    const CUtensorMap& im = *reinterpret_cast<const CUtensorMap*>(&in.m[i]);
    const CUtensorMap& om = *reinterpret_cast<const CUtensorMap*>(&out.m[i]);
    const CUtensorMap& rm = *reinterpret_cast<const CUtensorMap*>(res ? &res->m[i] : &out.m[i]);
    OB200_CUDA_OK(cudaLaunchKernelEx(&cfg, dtype == OB200_DTYPE_F16 ? conv_board8_kernel<true> : conv_board8_kernel<false>, im, om, rm, p));
    OB200_LAUNCHED("conv_board8_kernel");
    return OB200_OK;
}

// Blocks [part of 64 output channels][k_slice][dy] of 192 rows ([dx][output channel]) x 64 input channels, swizzled as
// conv_wide_pack's.  w: [cout][cin_real][9] fp32 (OIHW), scale: per output channel.
void conv_board8_pack(const float* w, const float* scale, int cout, int cin_real, int cin, void* packed_out, int dtype) {
    uint16_t* o = static_cast<uint16_t*>(packed_out);
    const int KS = cin / kSlice;
    for (int co = 0; co < cout; ++co)
        for (int ci = 0; ci < cin; ++ci)
            for (int tap = 0; tap < 9; ++tap) {
                const float v = ci < cin_real ? w[((size_t)co * cin_real + ci) * 9 + tap] * scale[co] : 0.0f;
                const int dy = tap / 3, row = tap % 3 * kNT + co % kNT, cil = ci % kSlice;
                const size_t block = ((size_t)(co / kNT) * KS + ci / kSlice) * 3 + dy;
                const size_t byte = block * kBStageBytes + (size_t)row * kRowBytes + (((cil >> 3) ^ (row & 7)) << 4) + (cil & 7) * 2;
                o[byte / 2] = dtype == OB200_DTYPE_F16 ? f32_to_f16_rne_sat(v) : f32_to_bf16_rne(v);
            }
}

}  // namespace ob200
