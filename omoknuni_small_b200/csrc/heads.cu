// Policy and value heads (sm_100a, fp32).
//
//   head_conv_kernel   1x1 convolution (+ folded BatchNorm, ReLU) of both heads
//                      from the tower's board tensor; writes fp32 activations
//                      in the reference's flatten order c * S*S + y * S + x
//                      (src/nn/resnet_model.cpp:183,209 view({B,-1}) on NCHW).
//   head_fc_kernel     the policy FC and the value head's first FC (head_fc.cu), tensor cores.
//   head_tails_kernel  their partial sums -> logits, softmax, value_fc2 + tanh, as one launch.
#include "internal.h"
#include "sm100_ptx.cuh"
#include "head_conv.cuh"
#include <algorithm>
#include <cmath>
#include <mutex>

namespace ob200 {
namespace {

using namespace ptx;

// A CTA takes tiles of 128 consecutive positions of the board tensor (pad positions included, their results are
// dropped): rows of 128 bytes per 64-channel slice into swizzled shared memory, two MMAs per 16 channels and slice
// (see head_conv.cuh; the same products in the same order as the board-resident tower's last layer), accumulators to
// the flattened head activations.  blockIdx.y: the group of up to 64 head channels.  HBM-bound for large batches (it
// reads the tower's output once per group): the next tile's rows are on their way into registers while a tile's MMAs
// and results are waited for, and several CTAs share an SM.  (2,048 boards of 19x19 x 128
// channels, 2 / 1 head channels: 54.8 us with the loads behind the MMAs, 40.6 now, 32 the bytes alone; 4,096 chess
// boards of 256 channels 58.1 -> 33.4; 512 boards of 19x19 x 128, 32 / 32 head channels, 45.1 -> 35.7.)
constexpr int kConvThreads = 256;
constexpr int kConvTile = 128;
constexpr int kConvTmemCols = 128;
struct HeadConvParams {
    const uint8_t* tower;
    HeadConvWeights head;
    float *hp, *hv;
    int hp_pitch, hv_pitch;
    int B, S, tiles;
    int* error;
};
// CTAs an SM: 128 TMEM columns and 16 registers a slice and thread for the rows under way each.
__host__ __device__ constexpr int conv_ctas_per_sm(int slices) { return slices == 1 ? 4 : slices == 2 ? 3 : 2; }
// SLICES: 64-channel slices of the tower.
template <bool F16, int SLICES>
__global__ void __launch_bounds__(kConvThreads, conv_ctas_per_sm(SLICES))
head_conv_kernel(const HeadConvParams p) {
    constexpr int kRowBytes = SLICES * 128, kVecs = SLICES * kConvTile * 8 / kConvThreads;     // 16-byte pieces a thread
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h0 = (int)blockIdx.y * 64, hc = min(64, p.head.hc - h0), rows = (hc + 15) / 16 * 16;
    uint8_t* a_s = smem;                                                // [slice][128 rows][128 bytes]
    uint8_t* w_s = smem + SLICES * kConvTile * 128;                     // [slice][split term][rows][128 bytes]
    const uint32_t w_bytes = (uint32_t)(SLICES * 3 * rows * 128);
    const uint32_t w_full = smem_u32(&bars[0]), done = smem_u32(&bars[1]);
    volatile int* abort_flag = &abort_s;
    if (threadIdx.x == 0) {
        mbar_init(w_full, 1); mbar_init(done, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_arrive_expect_tx(w_full, w_bytes);
        bulk_g2s(smem_u32(w_s), p.head.w + (size_t)blockIdx.y * SLICES * 3 * 64 * 128, w_bytes, w_full);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)kConvTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    OB200_PDL_ENTER();
    const int GP = p.S + 1, slots = GP * GP, S2 = p.S * p.S, total = p.B * slots;
    const uint32_t id2 = make_idesc(F16, kConvTile, 2 * rows), id1 = make_idesc(F16, kConvTile, rows);
    const int q = warp & 3, half = warp >> 2;
    uint32_t phase = 0;
    uint4 v[kVecs];
    auto fetch = [&](int tile) {          // the tensor is padded to whole tiles: every row is readable
        const uint8_t* src = p.tower + ((size_t)OB200_GUARD + (size_t)tile * kConvTile) * kRowBytes + threadIdx.x * 16;
#pragma unroll
        for (int j = 0; j < kVecs; ++j) v[j] = __ldcg(reinterpret_cast<const uint4*>(src + (size_t)j * (kConvThreads * 16)));
    };
    if ((int)blockIdx.x < p.tiles) fetch(blockIdx.x);
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, phase ^= 1u) {
#pragma unroll
        for (int j = 0; j < kVecs; ++j) {
            const int i = j * kConvThreads + threadIdx.x, c = i & 7, sl = (i >> 3) % SLICES, r = (i >> 3) / SLICES;
            *reinterpret_cast<uint4*>(a_s + (sl * kConvTile + r) * 128 + ((c ^ (r & 7)) << 4)) = v[j];
        }
        if (tile + (int)gridDim.x < p.tiles) fetch(tile + gridDim.x);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");    // the previous tile's accumulators have been read
        __syncthreads();
        if (threadIdx.x == 0) {
            if (mbar_wait(w_full, 0, abort_flag)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = desc_lo(smem_u32(a_s)), w = desc_lo(smem_u32(w_s));
                #pragma unroll
                for (int sl = 0; sl < SLICES; ++sl)
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        const uint32_t at = a + (uint32_t)(sl * kConvTile * 8 + ks * 2), wt = w + (uint32_t)(sl * 3 * rows * 8 + ks * 2);
                        umma(tmem_base, at, wt, id2, (sl | ks) ? 1u : 0u);
                        umma(tmem_base + (uint32_t)rows, at, wt + (uint32_t)(2 * rows * 8), id1, 1u);
                    }
                umma_commit(done);
            } else { abort_s = 1; atomicExch(p.error, 4); }
        }
        bool good = mbar_wait(done, phase, abort_flag);
        if (!__syncthreads_and(good)) { if (threadIdx.x == 0) atomicExch(p.error, 3); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int pos = tile * kConvTile + q * 32 + lane;
        const int b = pos / slots, r = pos - b * slots, y = r / GP, x = r - y * GP;
        const bool real = pos < total && y < p.S && x < p.S;
        const int cell = y * p.S + x;
        const uint32_t t = tmem_base + ((uint32_t)(q * 32) << 16);
        for (int c = half; c < rows / 8; c += 2) {
            uint32_t big[8], small[8];
            tmem_ld8(t + c * 8, big);
            tmem_ld8(t + rows + c * 8, small);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int h = h0 + c * 8 + j;
                if (c * 8 + j >= hc || !real) continue;
                const float o = head_conv_value(__uint_as_float(big[j]), __uint_as_float(small[j]), __ldg(p.head.scale + h), __ldg(p.head.bias + h));
                if (h < p.head.pc) p.hp[(size_t)b * p.hp_pitch + h * S2 + cell] = o;
                else p.hv[(size_t)b * p.hv_pitch + (h - p.head.pc) * S2 + cell] = o;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kConvTmemCols) : "memory");
}

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* red) {
    for (int off = 16; off > 0; off >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, v, off);
        v = is_max ? fmaxf(v, o) : v + o;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = red[0];
    for (int i = 1; i < nw; ++i) v = is_max ? fmaxf(v, red[i]) : v + red[i];
    return v;
}

constexpr int kTailThreads = 256;

// Elements j, j + kTailThreads, ... of row b of a layer's result (the first n of N exist): its slices of partial sums
// added in the layer's fixed order.  One element: fifteen loads (five groups of three, or fifteen groups) in flight at a
// time; four: six each.
template <int GROUP, int N>
__device__ __forceinline__ void sum_slices_in(const HeadFcLayer& l, const float* p, size_t step, int n, float (&total)[N]) {
    constexpr int kSliceBatch = N == 1 ? 15 : 6;
    static_assert(kSliceBatch % kHeadFcGroup == 0, "a batch of slices is a whole number of groups");
    for (int s = 0; s < l.slices; s += kSliceBatch) {
        float v[N][kSliceBatch];
#pragma unroll
        for (int e = 0; e < N; ++e)
#pragma unroll
            for (int k = 0; k < kSliceBatch; ++k)
                v[e][k] = s + k < l.slices && e < n ? __ldcg(p + (size_t)(s + k) * step + e * kTailThreads) : 0.0f;
#pragma unroll
        for (int g = 0; g < kSliceBatch; g += GROUP) {
            if (s + g >= l.slices) break;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                float group = v[e][g];
#pragma unroll
                for (int k = g + 1; k < g + GROUP; ++k)
                    if (s + k < l.slices) group = __fadd_rn(group, v[e][k]);
                total[e] = s + g ? __fadd_rn(total[e], group) : group;
            }
        }
    }
}
template <int N>
__device__ __forceinline__ void sum_slices(const HeadFcLayer& l, int b, int B, int j, int n, float (&total)[N]) {
    const float* p = l.part + (size_t)b * l.part_pitch + j;
    const size_t step = (size_t)B * l.part_pitch;
    if (l.slices == 1) {
#pragma unroll
        for (int e = 0; e < N; ++e) total[e] = e < n ? __ldcg(p + e * kTailThreads) : 0.0f;
    } else if (l.slice_group == 1) sum_slices_in<1, N>(l, p, step, n, total);
    else sum_slices_in<kHeadFcGroup, N>(l, p, step, n, total);
}
__device__ __forceinline__ float sum_slices(const HeadFcLayer& l, int b, int B, int j) {
    float total[1];
    sum_slices(l, b, B, j, 1, total);
    return total[0];
}

// The tails of both heads in one launch, started as a programmatic dependent of the FC kernel: CTAs [0, policy_ctas)
// finish a row of logits each (sum of the slices, bias, softmax: maximum, sum of exponentials, division), or a share of a
// long one that is not normalised, the rest one board's value each.  A thread per output: what a small batch waits for is
// the trip to L2 for the slices, so a thread of a longer row sums four outputs at a time and long rows of plain logits are
// shared out.  4,672 logits of one board, an evaluation: 450 terms 46.7 us with one output at a time, 38.6 with four, 32.9
// shared out as well; 128 terms 33.0, 30.6, 26.7.
constexpr int kTailRegs = 2;             // logits a thread keeps in registers: rows of up to 512
constexpr int kTailAhead = 4;            // outputs a thread of a longer row sums at a time
constexpr int kTailSpan = kTailAhead * kTailThreads;     // a CTA's share of a longer row that is not normalised
__global__ void __launch_bounds__(kTailThreads)
head_tails_kernel(const HeadFcLayer pol, const float* __restrict__ bp, float* __restrict__ logits, int A, int policy_ctas, int row_parts, int softmax,
                  const HeadFcLayer val, const float* __restrict__ b1, const float* __restrict__ w2, float b2, int H, int B,
                  float* __restrict__ value, const int* error_word, int* error_out) {
    __shared__ float red[kTailThreads / 32];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (error_out && blockIdx.x == 0 && threadIdx.x == 0) *error_out = __ldcg(error_word);
    if ((int)blockIdx.x < policy_ctas) {
        const int b = (int)blockIdx.x / row_parts;
        float* row = logits + (size_t)b * A;
        if (A <= kTailRegs * kTailThreads) {
            float x[kTailRegs];
            float m = -INFINITY;
#pragma unroll
            for (int k = 0; k < kTailRegs; ++k) {
                const int i = threadIdx.x + k * kTailThreads;
                x[k] = -INFINITY;
                if (i < A) x[k] = pol.part ? __fadd_rn(sum_slices(pol, b, B, i), bp[i]) : row[i];
                m = fmaxf(m, x[k]);
            }
            float scale = 1.0f;
            if (softmax) {
                m = block_reduce(m, true, red);
                float s = 0.0f;
#pragma unroll
                for (int k = 0; k < kTailRegs; ++k)
                    if ((int)threadIdx.x + k * kTailThreads < A) { x[k] = expf(x[k] - m); s += x[k]; }
                scale = 1.0f / block_reduce(s, false, red);
            }
#pragma unroll
            for (int k = 0; k < kTailRegs; ++k) {
                const int i = threadIdx.x + k * kTailThreads;
                if (i < A) row[i] = x[k] * scale;
            }
            return;
        }
        float m = -INFINITY;
        const int from = ((int)blockIdx.x - b * row_parts) * kTailSpan, to = row_parts > 1 ? min(A, from + kTailSpan) : A;
        for (int i0 = from + threadIdx.x; i0 < to; i0 += kTailSpan) {
            const int n = (A - i0 + kTailThreads - 1) / kTailThreads;
            float x[kTailAhead];
            if (pol.part) sum_slices(pol, b, B, i0, n, x);
#pragma unroll
            for (int k = 0; k < kTailAhead; ++k) {
                if (k >= n) break;
                const int i = i0 + k * kTailThreads;
                if (pol.part) row[i] = x[k] = __fadd_rn(x[k], bp[i]);
                else x[k] = row[i];
                m = fmaxf(m, x[k]);
            }
        }
        if (!softmax) return;
        m = block_reduce(m, true, red);
        float s = 0.0f;
        for (int i = threadIdx.x; i < A; i += kTailThreads) s += expf(row[i] - m);
        s = block_reduce(s, false, red);
        const float inv = 1.0f / s;
        for (int i = threadIdx.x; i < A; i += kTailThreads) row[i] = expf(row[i] - m) * inv;
    } else {
        const int b = (int)blockIdx.x - policy_ctas;
        float s = 0.0f;
        for (int i = threadIdx.x; i < H; i += kTailThreads) s = fmaf(relu_keep_nan(__fadd_rn(sum_slices(val, b, B, i), b1[i])), w2[i], s);
        s = block_reduce(s, false, red);
        if (threadIdx.x == 0) value[b] = tanhf(s + b2);
    }
}

}  // namespace

int launch_head_tails(const HeadFcLayer& policy, const float* bp, float* policy_out, int policy_size, int softmax,
                      const HeadFcLayer& value, const float* b1, int H, const float* w2, float b2, float* value_out, int B,
                      cudaStream_t st, int* error_out) {
    const int rows = policy_out && (policy.part || softmax) ? B : 0;
    const int parts = softmax || policy_size <= kTailRegs * kTailThreads ? 1 : (policy_size + kTailSpan - 1) / kTailSpan;
    OB200_CUDA_OK(launch_dependent(head_tails_kernel, dim3((unsigned)(rows * parts + B)), dim3(kTailThreads), 0, st, policy, bp,
                                   policy_out, policy_size, rows * parts, parts, softmax, value, b1, w2, b2, H, B, value_out,
                                   (const int*)(error_out ? device_error_word() : nullptr), error_out));
    counters().launches.fetch_add(1, std::memory_order_relaxed);
    return OB200_OK;
}

size_t head_conv_packed_bytes(int hc, int C) {
    const int last = hc % 64, rows = hc / 64 * 64 + (last + 15) / 16 * 16;
    return (size_t)rows * 3 * C * 2;
}

void head_conv_pack(const float* w, int hc, int C, int dtype, void* packed_out, float* scale_out) {
    std::memset(packed_out, 0, head_conv_packed_bytes(hc, C));
    const int slices = C / 64;
    for (int h = 0; h < hc; ++h) {
        const int group = h / 64, row = h % 64, in_group = hc - group * 64 < 64 ? hc - group * 64 : 64, rows = (in_group + 15) / 16 * 16;
        // fp16: bring the channel's largest weight to [2^12, 2^13), a power of two that the result is divided by
        float up = 1.0f;
        if (dtype == OB200_DTYPE_F16) {
            float top = 0.0f;
            for (int k = 0; k < C; ++k) top = std::max(top, std::fabs(w[(size_t)h * C + k]));
            int e = 0;
            if (top > 0.0f && std::isfinite(top)) { std::frexp(top, &e); up = std::ldexp(1.0f, std::min(13 - e, 100)); }
        }
        scale_out[h] = 1.0f / up;
        for (int k = 0; k < C; ++k) {
            float v = w[(size_t)h * C + k] * up;
            uint8_t* at = static_cast<uint8_t*>(packed_out) + ((size_t)group * slices * 64 + (size_t)(k / 64) * rows) * 3 * 128 + row * 128 +
                          ((((k & 63) >> 3) ^ (row & 7)) << 4) + (k & 7) * 2;
            for (int t = 0; t < 3; ++t) {
                uint16_t u;
                float f;
                uint32_t bits;
                std::memcpy(&bits, &v, 4);
                if (dtype == OB200_DTYPE_F16) {
                    // an infinite weight stays one
                    u = std::isinf(v) ? (uint16_t)(((bits >> 16) & 0x8000u) | 0x7C00u) : f32_to_f16_rne_sat(v);
                    f = __half2float(*reinterpret_cast<const __half*>(&u));
                } else {
                    u = f32_to_bf16_rne(v);
                    if ((u & 0x7FFFu) == 0x7F80u) u = (uint16_t)(bits >> 16);      // a finite one does not become one
                    const uint32_t b = (uint32_t)u << 16;
                    std::memcpy(&f, &b, 4);
                }
                std::memcpy(at + (size_t)t * rows * 128, &u, 2);
                if (!std::isfinite(v)) break;                                       // no lower terms
                v -= f;
            }
        }
    }
}

int launch_head_conv(const void* tower, const HeadConvWeights& head, float* hp, float* hv, int hp_pitch, int hv_pitch, int B, int S,
                     cudaStream_t st, int C, int dtype) {
    if (C < 64 || C % 64 || C > 256 || head.hc < 1)
        return set_error(OB200_ERR_INVALID, "head conv: tower channels %d not a multiple of 64 up to 256, or no head channels", C);
    if (int rc = require_device()) return rc;
    int dev = 0, sms = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    OB200_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const BoardGeom g = board_geom(S, B);
    if (g.P > 0x7fffffffLL - kConvTile) return set_error(OB200_ERR_TOO_LARGE, "head conv: batch too large");
    HeadConvParams p;
    p.tower = static_cast<const uint8_t*>(tower); p.head = head; p.hp = hp; p.hv = hv; p.hp_pitch = hp_pitch; p.hv_pitch = hv_pitch;
    p.B = B; p.S = S; p.tiles = (int)(g.Ppad / kConvTile);
    p.error = device_error_word();
    if (!p.error) return set_error(OB200_ERR_CUDA, "head conv: cannot resolve the device error word");
    const int groups = (head.hc + 63) / 64, rows = (std::min(head.hc, 64) + 15) / 16 * 16;
    const int slices = C / 64;
    const size_t smem = (size_t)slices * (kConvTile + 3 * rows) * 128 + 1024;
    using Kernel = void (*)(HeadConvParams);
    static const Kernel kernels[2][4] = {
        {head_conv_kernel<false, 1>, head_conv_kernel<false, 2>, head_conv_kernel<false, 3>, head_conv_kernel<false, 4>},
        {head_conv_kernel<true, 1>, head_conv_kernel<true, 2>, head_conv_kernel<true, 3>, head_conv_kernel<true, 4>}};
    const int f16 = dtype == OB200_DTYPE_F16;
    const Kernel kernel = kernels[f16][slices - 1];
    static bool configured[64][2][4] = {};
    if (dev < 0 || dev >= 64 || !configured[dev][f16][slices - 1]) {
        OB200_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, slices * (kConvTile + 3 * 64) * 128 + 1024));
        if (dev >= 0 && dev < 64) configured[dev][f16][slices - 1] = true;
    }
    // as many CTAs an SM as their shared memory leaves room for
    const int per_sm = std::max(1, std::min(conv_ctas_per_sm(slices), (int)(220 * 1024 / (smem + 1024))));
    OB200_CUDA_OK(launch_dependent(kernel, dim3(std::min(p.tiles, sms * per_sm), groups), dim3(kConvThreads), smem, st, p));
    counters().launches.fetch_add(1, std::memory_order_relaxed);
    return OB200_OK;
}

// ---------------------------------------------------------------------------
// Value head without any allocation.  The two intermediates of the value head
// (the 1x1-convolution activations and the hidden layer) live in this
// file-scope device array instead of buffers obtained from cudaMalloc.  Every
// GPU that loads the library holds the 2 MiB until the process exits.
// ---------------------------------------------------------------------------
constexpr size_t kStaticScratchFloats = size_t(1) << 19;
static __device__ __align__(256) float g_value_head_scratch[kStaticScratchFloats];

size_t value_head_static_capacity() { return kStaticScratchFloats; }

// In host code the array's name is only a stand-in for the symbol: its device address
// is asked from the runtime once per device, with that device current.
static int value_head_scratch_ptr(float** out) {
    static std::mutex mu;
    static float* cached[64] = {nullptr};
    int dev = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_error(OB200_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (!cached[dev]) {
        void* ptr = nullptr;
        OB200_CUDA_OK(cudaGetSymbolAddress(&ptr, g_value_head_scratch));
        cached[dev] = static_cast<float*>(ptr);
    }
    *out = cached[dev];
    return OB200_OK;
}

int launch_value_head_static(const void* tower, const HeadConvWeights& value_conv, const HeadFcLayer& value_layer,
                             const float* b1, const float* w2, float b2, int H, int B, int S, float* value_out,
                             cudaStream_t st, int dtype) {
    const int vc = value_conv.hc;
    const size_t need = (size_t)B * ((size_t)vc * S * S + (size_t)H);
    if (need > kStaticScratchFloats)
        return set_error(OB200_ERR_TOO_LARGE,
                         "value head without allocation: batch %d needs %zu scratch floats (%d x %d x %d + %d per board), the static array holds %zu",
                         B, need, vc, S, S, H, kStaticScratchFloats);
    float* scratch = nullptr;
    if (int rc = value_head_scratch_ptr(&scratch)) return rc;
    // Rows of a multiple of four floats, which the FC kernel reads and writes 16 bytes at a time, and the layer's chunks
    // spread over CTAs as a forward spreads them, where the scratch holds that; rows as they are and all chunks in one CTA
    // per tile otherwise.  Either way every element read below is written first by the launch before it, or cleared (inputs
    // beyond K): nothing needs clearing here.  (15x15, one value channel: 149 boards 33 us with rows as they
    // are and all chunks in one CTA, 19 so; 300 boards 29 / 19; 30x30, 64 boards 47 / 17.)
    HeadFcLayer l = value_layer;
    int dev = 0, sms = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    OB200_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int K = vc * S * S;
    l.in_pitch = (K + 3) / 4 * 4; l.part_pitch = (H + 3) / 4 * 4;
    head_fc_plan(&l, 1, B, sms);
    auto fits = [&]() { return (size_t)B * ((size_t)l.in_pitch + (size_t)l.slices * l.part_pitch) <= kStaticScratchFloats; };
    if (!fits() && l.chunks_per_slice == 1) { l.chunks_per_slice = kHeadFcGroup; l.slices = (l.chunks + kHeadFcGroup - 1) / kHeadFcGroup; l.slice_group = 1; }
    if (!fits()) { l.chunks_per_slice = l.chunks; l.slices = 1; l.slice_group = 1; }
    if (!fits()) { l.in_pitch = K; l.part_pitch = H; }
    float* hv = scratch;                                  // [B][in_pitch]
    l.in = hv; l.part = scratch + (size_t)B * l.in_pitch; // [slice][B][part_pitch]
    if (int rc = launch_head_conv(tower, value_conv, nullptr, hv, 0, l.in_pitch, B, S, st, 64, dtype)) return rc;
    if (int rc = launch_head_fc(&l, 1, B, st)) return rc;
    return launch_head_tails(HeadFcLayer{}, nullptr, nullptr, 0, 0, l, b1, H, w2, b2, value_out, B, st);
}

}  // namespace ob200
