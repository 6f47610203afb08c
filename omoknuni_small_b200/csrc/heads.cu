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
#include <mutex>

namespace ob200 {
namespace {

struct alignas(16) Pack8 { uint32_t v[4]; };

// A warp takes 32 consecutive positions of the board tensor (pad positions included, their
// results are dropped).  Eight lanes share a position: lane = 8 * (position within a group of 4)
// + channel block, so a warp-wide 16-byte load covers 4 positions x 128 contiguous bytes of one
// 64-channel slice and the 8 loads of a warp are issued back to back.  Each lane multiplies its
// 8 channels (per slice) into a head channel's partial sum, three shuffle steps add the 8 lanes,
// and lane (sub, blk) keeps the sum of group blk: after 8 groups every lane owns one position and
// stores once per head channel.  C = tower channels (a multiple of 64).
// HCT > 0: that many head channels, partial sums of all of them held in registers while the
// slices stream by; HCT == 0: any number, weights in shared memory, one head channel at a time.
constexpr int kHeadThreads = 128;
template <int HCT>
__global__ void __launch_bounds__(kHeadThreads)
head_conv_kernel(const uint8_t* __restrict__ tower, const float* __restrict__ w,
                 const float* __restrict__ bias, int HC, int pc, float* __restrict__ hp,
                 float* __restrict__ hv, int hp_pitch, int hv_pitch, int B, int S, int C, int f16) {
    extern __shared__ float w_s[];  // HCT == 0: [HC][C] folded weights then [HC] biases
    const int lane = threadIdx.x & 31, sub = lane >> 3, blk = lane & 7;
    if (HCT == 0) {
        for (int i = threadIdx.x; i < HC * C; i += blockDim.x) w_s[i] = w[i];
        for (int i = threadIdx.x; i < HC; i += blockDim.x) w_s[HC * C + i] = bias[i];
        __syncthreads();
    }
    const int hc = HCT > 0 ? HCT : HC;
    const int S2 = S * S, GP = S + 1, slots = GP * GP;
    const int total = B * slots;
    const int slices = C >> 6;
    const size_t row_bytes = (size_t)C * 2;
    const int p0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
    if (p0 >= total) return;
    // the tensor's trailing guard positions make the (at most 31) positions past the end readable
    const uint8_t* src = tower + ((size_t)OB200_GUARD + p0 + sub) * row_bytes + blk * 16;
    float a[8][8];
    auto load_slice = [&](int sl) {
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const Pack8 v = *reinterpret_cast<const Pack8*>(src + (size_t)it * 4 * row_bytes + (size_t)sl * 128);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // the tower's storage type: both conversions are exact
                if (f16) ptx::unpack2<true>(v.v[j], a[it][2 * j], a[it][2 * j + 1]);
                else ptx::unpack2<false>(v.v[j], a[it][2 * j], a[it][2 * j + 1]);
            }
        }
    };
    // this lane's own position: group blk, member sub
    const int p = p0 + blk * 4 + sub;
    const int b = p / slots, r = p - b * slots;
    const int y = r / GP, x = r - y * GP;
    const bool real = p < total && y < S && x < S;
    const int cell = y * S + x;
    auto finish = [&](int h, const float (&part)[8], float bh) {
        float keep = 0.0f;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            float s = part[it];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            keep = (it == blk) ? s : keep;
        }
        if (real) {
            const float o = fmaxf(keep + bh, 0.0f);
            if (h < pc) hp[(size_t)b * hp_pitch + h * S2 + cell] = o;
            else hv[(size_t)b * hv_pitch + (h - pc) * S2 + cell] = o;
        }
    };
    if (HCT > 0) {
        constexpr int kRegCh = HCT > 0 ? HCT : 1;
        float part[kRegCh][8];
#pragma unroll
        for (int h = 0; h < kRegCh; ++h)
#pragma unroll
            for (int it = 0; it < 8; ++it) part[h][it] = 0.0f;
        for (int sl = 0; sl < slices; ++sl) {
            load_slice(sl);
#pragma unroll
            for (int h = 0; h < kRegCh; ++h) {
                const float4* wr = reinterpret_cast<const float4*>(w + (size_t)h * C + sl * 64 + blk * 8);
                const float4 w0 = __ldg(wr), w1 = __ldg(wr + 1);
                const float wk[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int it = 0; it < 8; ++it)
#pragma unroll
                    for (int k = 0; k < 8; ++k) part[h][it] = fmaf(a[it][k], wk[k], part[h][it]);
            }
        }
#pragma unroll
        for (int h = 0; h < kRegCh; ++h) finish(h, part[h], __ldg(bias + h));
    } else {
        if (slices == 1) load_slice(0);
        for (int h = 0; h < hc; ++h) {
            float part[8];
#pragma unroll
            for (int it = 0; it < 8; ++it) part[it] = 0.0f;
            for (int sl = 0; sl < slices; ++sl) {
                if (slices > 1) load_slice(sl);   // re-read per head channel (L1 / L2 hits)
                const float4* wr = reinterpret_cast<const float4*>(w_s + (size_t)h * C + sl * 64 + blk * 8);
                const float4 w0 = wr[0], w1 = wr[1];
                const float wk[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int it = 0; it < 8; ++it)
#pragma unroll
                    for (int k = 0; k < 8; ++k) part[it] = fmaf(a[it][k], wk[k], part[it]);
            }
            finish(h, part, w_s[hc * C + h]);
        }
    }
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

// Element j of row b of a layer's result: its slices of partial sums added in the layer's fixed order, fifteen loads
// (five groups of three, or fifteen groups) in flight at a time.
constexpr int kSliceBatch = 15;
static_assert(kSliceBatch % kHeadFcGroup == 0, "a batch of slices is a whole number of groups");
template <int GROUP>
__device__ __forceinline__ float sum_slices_in(const HeadFcLayer& l, const float* p, size_t step) {
    float total = 0.0f;
    for (int s = 0; s < l.slices; s += kSliceBatch) {
        float v[kSliceBatch];
#pragma unroll
        for (int k = 0; k < kSliceBatch; ++k) v[k] = s + k < l.slices ? __ldcg(p + (size_t)(s + k) * step) : 0.0f;
#pragma unroll
        for (int g = 0; g < kSliceBatch; g += GROUP) {
            if (s + g >= l.slices) break;
            float group = v[g];
#pragma unroll
            for (int k = g + 1; k < g + GROUP; ++k)
                if (s + k < l.slices) group = __fadd_rn(group, v[k]);
            total = s + g ? __fadd_rn(total, group) : group;
        }
    }
    return total;
}
__device__ __forceinline__ float sum_slices(const HeadFcLayer& l, int b, int B, int j) {
    const float* p = l.part + (size_t)b * l.part_pitch + j;
    const size_t step = (size_t)B * l.part_pitch;
    if (l.slices == 1) return __ldcg(p);
    return l.slice_group == 1 ? sum_slices_in<1>(l, p, step) : sum_slices_in<kHeadFcGroup>(l, p, step);
}

// The tails of both heads in one launch, started as a programmatic dependent of the FC kernel: CTAs [0, policy_rows)
// finish one row of logits each (sum of the slices, bias, softmax: maximum, sum of exponentials, division), the rest
// one board's value each.  A thread per output: what a small batch waits for is the trip to L2 for the slices.
constexpr int kTailThreads = 256;
constexpr int kTailRegs = 2;             // logits a thread keeps in registers: rows of up to 512
__global__ void __launch_bounds__(kTailThreads)
head_tails_kernel(const HeadFcLayer pol, const float* __restrict__ bp, float* __restrict__ logits, int A, int policy_rows, int softmax,
                  const HeadFcLayer val, const float* __restrict__ b1, const float* __restrict__ w2, float b2, int H, int B,
                  float* __restrict__ value) {
    __shared__ float red[kTailThreads / 32];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if ((int)blockIdx.x < policy_rows) {
        const int b = blockIdx.x;
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
        for (int i = threadIdx.x; i < A; i += kTailThreads) {
            if (pol.part) row[i] = __fadd_rn(sum_slices(pol, b, B, i), bp[i]);
            m = fmaxf(m, row[i]);
        }
        if (!softmax) return;
        m = block_reduce(m, true, red);
        float s = 0.0f;
        for (int i = threadIdx.x; i < A; i += kTailThreads) s += expf(row[i] - m);
        s = block_reduce(s, false, red);
        const float inv = 1.0f / s;
        for (int i = threadIdx.x; i < A; i += kTailThreads) row[i] = expf(row[i] - m) * inv;
    } else {
        const int b = (int)blockIdx.x - policy_rows;
        float s = 0.0f;
        for (int i = threadIdx.x; i < H; i += kTailThreads) s = fmaf(fmaxf(__fadd_rn(sum_slices(val, b, B, i), b1[i]), 0.0f), w2[i], s);
        s = block_reduce(s, false, red);
        if (threadIdx.x == 0) value[b] = tanhf(s + b2);
    }
}

}  // namespace

int launch_head_tails(const HeadFcLayer& policy, const float* bp, float* policy_out, int policy_size, int softmax,
                      const HeadFcLayer& value, const float* b1, int H, const float* w2, float b2, float* value_out, int B,
                      cudaStream_t st) {
    const int rows = policy_out && (policy.part || softmax) ? B : 0;
    OB200_CUDA_OK(launch_dependent(head_tails_kernel, dim3((unsigned)(rows + B)), dim3(kTailThreads), 0, st, policy, bp,
                                   policy_out, policy_size, rows, softmax, value, b1, w2, b2, H, B, value_out));
    counters().launches.fetch_add(1, std::memory_order_relaxed);
    return OB200_OK;
}

int launch_head_conv(const void* tower, const float* w, const float* bias, int HC, int pc,
                     float* hp, float* hv, int hp_pitch, int hv_pitch, int B, int S, cudaStream_t st, int C, int dtype) {
    const int f16 = dtype == OB200_DTYPE_F16;
    if (C < 64 || C % 64) return set_error(OB200_ERR_INVALID, "head conv: tower channels %d not a multiple of 64", C);
    const long long total = (long long)B * (S + 1) * (S + 1);   // positions, one warp per 32
    const unsigned grid = (unsigned)((total + kHeadThreads - 1) / kHeadThreads);
    const uint8_t* t = static_cast<const uint8_t*>(tower);
    switch (HC) {
        case 1: head_conv_kernel<1><<<grid, kHeadThreads, 0, st>>>(t, w, bias, HC, pc, hp, hv, hp_pitch, hv_pitch, B, S, C, f16); break;
        case 2: head_conv_kernel<2><<<grid, kHeadThreads, 0, st>>>(t, w, bias, HC, pc, hp, hv, hp_pitch, hv_pitch, B, S, C, f16); break;
        case 3: head_conv_kernel<3><<<grid, kHeadThreads, 0, st>>>(t, w, bias, HC, pc, hp, hv, hp_pitch, hv_pitch, B, S, C, f16); break;
        case 4: head_conv_kernel<4><<<grid, kHeadThreads, 0, st>>>(t, w, bias, HC, pc, hp, hv, hp_pitch, hv_pitch, B, S, C, f16); break;
        default: {
            const size_t smem = (size_t)(HC * C + HC) * sizeof(float);
            if (smem > 200 * 1024)
                return set_error(OB200_ERR_UNSUPPORTED, "head conv: %d head channels x %d tower channels exceed shared memory", HC, C);
            if (smem > 48 * 1024)
                OB200_CUDA_OK(cudaFuncSetAttribute(head_conv_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            head_conv_kernel<0><<<grid, kHeadThreads, smem, st>>>(t, w, bias, HC, pc, hp, hv, hp_pitch, hv_pitch, B, S, C, f16);
        }
    }
    OB200_LAUNCHED("head_conv_kernel");
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

int launch_value_head_static(const void* tower, const float* vw, const float* vb, int vc, const HeadFcLayer& value_layer,
                             const float* b1, const float* w2, float b2, int H, int B, int S, float* value_out,
                             cudaStream_t st, int dtype) {
    const size_t need = (size_t)B * ((size_t)vc * S * S + (size_t)H);
    if (need > kStaticScratchFloats)
        return set_error(OB200_ERR_TOO_LARGE,
                         "value head without allocation: batch %d needs %zu scratch floats (%d x %d x %d + %d per board), the static array holds %zu",
                         B, need, vc, S, S, H, kStaticScratchFloats);
    float* scratch = nullptr;
    if (int rc = value_head_scratch_ptr(&scratch)) return rc;
    float* hv = scratch;                                  // [B][vc * S * S]
    float* hidden = scratch + (size_t)B * vc * S * S;     // [B][H]
    // every element read below is written first by the launch before it: nothing needs clearing
    if (int rc = launch_head_conv(tower, vw, vb, vc, 0, hv, hv, 0, vc * S * S, B, S, st, 64, dtype)) return rc;
    // the layer with all its chunks in one CTA per tile: one slice, which fits the scratch
    HeadFcLayer l = value_layer;
    l.in = hv; l.in_pitch = vc * S * S; l.part = hidden; l.part_pitch = H;
    l.chunks_per_slice = l.chunks; l.slices = 1; l.slice_group = 1;
    if (int rc = launch_head_fc(&l, 1, B, st)) return rc;
    return launch_head_tails(HeadFcLayer{}, nullptr, nullptr, 0, 0, l, b1, H, w2, b2, value_out, B, st);
}

}  // namespace ob200
