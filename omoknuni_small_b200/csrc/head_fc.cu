// The fully connected layers of both heads on the tensor cores, in fp32 precision (sm_100a).
//
// out[b][j] = sum_k in[b][k] * w[j][k] with fp32 inputs and weights.  tcgen05.mma takes 16-bit operands, so both
// operands are split exactly into three bf16 terms (x = x0 + x1 + x2: 8 + 8 + 8 significant bits hold fp32's 24)
// and six of the nine products are summed in fp32: x0w0, x0w1, x1w0, x1w1, x0w2, x2w0.  The three left out are below
// 2^-25 of |x||w|, half a unit in the last place of the product.  The tensor core's accumulator rounds less well than
// an fp32 addition, so sums in it are kept short and unlike terms apart: x0w0 has an accumulator of its own (with all
// six products in one, the logits of the 32-channel heads were 1.3e-6 from an fp64 evaluation, 2-norm, against 0.8e-6
// for a chain of fp32 multiply-adds; apart, 0.14e-6), it covers one CHUNK of the inner dimension (128 or 256 terms),
// chunks are added in fp32 in groups of three, and the groups in order.  That order depends on the layer alone, never
// on the batch or on which CTA computes what, so a position's result does not depend on the batch it comes in.
//
// A CTA owns 128 boards x 128 outputs and a run of chunks: one chunk (small batches: the chunks of the inner
// dimension are what there is to spread over the SMs), one group, or all of them (large batches).  Its sums leave as
// one slice of partial sums; head_tails_kernel (heads.cu) adds the slices in the fixed order.
//   * Weights are split, swizzled and laid out once, in the order they are read: a stage of 32 inner terms
//     (3 x 128 x 64 bytes) is one bulk copy.  Four stages of 48 KB (weights 24 KB, inputs 24 KB).
//   * Inputs are fp32 in memory; eight warps load them two stages ahead, split them in registers and store the three
//     swizzled tiles.  The same warps drain a chunk's accumulators while the next chunk's MMAs run (two accumulators).
//   * One thread issues the MMAs: 12 of 128x128x16 a stage = 768 cycles.
// What bounds it: small batches, the chain load -> split -> 8 stages of MMAs -> drain; large ones, the stages' 40 KB
// from L2 per 768 cycles (52 bytes a cycle and SM).  A whole evaluation through host buffers, 32 / 32-channel heads
// (7,200 terms), with the register-tiled fp32 kernel this one replaces and now: 1 board 368 -> 143 us, 250 boards 439
// -> 221 us (that kernel took 236 us for either: eight CTAs' worth of a serial loop over 7,200 terms).
#include "internal.h"
#include "sm100_ptx.cuh"
#include <cfloat>

namespace ob200 {
namespace {

using namespace ptx;

constexpr int kM = 128, kN = 128, kStageK = 32;
constexpr int kRowBytes = kStageK * 2;
constexpr int kTileBytes = 128 * kRowBytes;              // 8,192: one split term of one operand
constexpr int kOperandBytes = 3 * kTileBytes;
constexpr int kStageBytes = 2 * kOperandBytes;           // inputs, then weights
constexpr int kStages = 4;
constexpr int kSplitWarps = 8;
constexpr int kThreads = 32 * (kSplitWarps + 2);         // warps 0-7: split + drain, 8: weight loader, 9: MMA issue
constexpr int kTmemCols = 4 * kN;                       // two chunks x (large products, small products)
constexpr int kNumBars = 3 * kStages + 4;
constexpr int kSmemBytes = kStages * kStageBytes + kNumBars * 8 + 16 + 1024;

struct SplitParams {
    HeadFcLayer layer[2];
    int entries0;             // blockIdx.y values that belong to layer 0
    int B;
    int* error;
};

// x0, x1 -> three words of two bf16 terms each (low half: x0's).
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack2<false>(x0, x1);
    float a, b;
    unpack2<false>(h, a, b);
    x0 = __fsub_rn(x0, a); x1 = __fsub_rn(x1, b);        // exact
    m = pack2<false>(x0, x1);
    unpack2<false>(m, a, b);
    l = pack2<false>(__fsub_rn(x0, a), __fsub_rn(x1, b));
}

// VEC: the layers' input rows are 16-byte aligned (their padding, up to a multiple of four floats, holds finite values).
template <bool VEC>
__global__ void __launch_bounds__(kThreads, 1)
head_fc_kernel(const SplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar0 = smem_u32(bars);
    auto in_full = [&](int s) { return bar0 + 8u * s; };
    auto w_full = [&](int s) { return bar0 + 8u * (kStages + s); };
    auto empty = [&](int s) { return bar0 + 8u * (2 * kStages + s); };
    auto acc_full = [&](int a) { return bar0 + 8u * (3 * kStages + a); };
    auto acc_empty = [&](int a) { return bar0 + 8u * (3 * kStages + 2 + a); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(in_full(s), kSplitWarps); mbar_init(w_full(s), 1); mbar_init(empty(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), kSplitWarps); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    // this CTA's layer, output tile and run of chunks
    const bool second = (int)blockIdx.y >= p.entries0;
    HeadFcLayer L = p.layer[0];          // (a run-time index into the parameters would put every use of them in local memory)
    if (second) L = p.layer[1];
    const int entry = (int)blockIdx.y - (second ? p.entries0 : 0);
    const int tile_n = entry % L.n_tiles, slice = entry / L.n_tiles;
    const int chunk0 = slice * L.chunks_per_slice, chunk1 = min(L.chunks, chunk0 + L.chunks_per_slice);
    const int stages_per_chunk = L.chunk_k / kStageK;
    const int kb0 = chunk0 * stages_per_chunk, kb1 = min(L.k_blocks, chunk1 * stages_per_chunk);
    const int n_stages = kb1 - kb0;

    if (warp == 8) {
        // ---------------- weights: constants of the network, no need to wait for the kernel ahead ----------------
        if (lane == 0) {
            const uint8_t* src = L.w + ((size_t)tile_n * L.k_blocks + kb0) * kOperandBytes;
            bool ok = true;
            for (int i = 0; i < n_stages; ++i) {
                const int s = i % kStages;
                if (!mbar_wait(empty(s), ((uint32_t)(i / kStages) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                mbar_arrive_expect_tx(w_full(s), (uint32_t)kOperandBytes);
                bulk_g2s(smem_u32(smem + s * kStageBytes + kOperandBytes), src + (size_t)i * kOperandBytes, (uint32_t)kOperandBytes, w_full(s));
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.error, 4); }
        }
    } else if (warp == 9) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            constexpr uint32_t kIdesc = make_idesc(false, kM, kN);
            constexpr int kTile = kTileBytes >> 4;
            bool ok = true;
            int i = 0;
            for (int c = chunk0; ok && c < chunk1; ++c) {
                const int acc = (c - chunk0) & 1;
                if (!mbar_wait(acc_empty(acc), ((uint32_t)((c - chunk0) >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                const uint32_t d = tmem_base + (uint32_t)(acc * 2 * kN), d_small = d + kN;
                const int last = min(n_stages, (c + 1 - chunk0) * stages_per_chunk);
                bool first = true;
                for (; i < last; ++i) {
                    const int s = i % kStages;
                    const uint32_t ph = (uint32_t)(i / kStages) & 1u;
                    if (!mbar_wait(w_full(s), ph, abort_flag) || !mbar_wait(in_full(s), ph, abort_flag)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a = desc_lo(smem_u32(smem + s * kStageBytes)), b = desc_lo(smem_u32(smem + s * kStageBytes + kOperandBytes));
#pragma unroll
                    for (int ks = 0; ks < kStageK / 16; ++ks) {
                        const uint32_t more = (first && ks == 0) ? 0u : 1u;
                        umma<kDescHi64>(d_small, a + 2 * kTile + ks * 2, b + ks * 2, kIdesc, more);
                        umma<kDescHi64>(d_small, a + ks * 2, b + 2 * kTile + ks * 2, kIdesc, 1u);
                        umma<kDescHi64>(d_small, a + kTile + ks * 2, b + kTile + ks * 2, kIdesc, 1u);
                        umma<kDescHi64>(d_small, a + kTile + ks * 2, b + ks * 2, kIdesc, 1u);
                        umma<kDescHi64>(d_small, a + ks * 2, b + kTile + ks * 2, kIdesc, 1u);
                        umma<kDescHi64>(d, a + ks * 2, b + ks * 2, kIdesc, more);
                    }
                    first = false;
                    umma_commit(empty(s));
                }
                if (ok) umma_commit(acc_full(acc));
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.error, 2); }
        }
    } else {
        // ---------------- inputs -> three bf16 tiles; accumulators -> sums ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");               // the inputs come from the kernel ahead in the stream
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        const int row0 = (int)blockIdx.x * kM;
        const int sub = lane >> 3, kv = (lane & 7) * 4;                  // four rows a step, eight float4 a row
        float4 xs[2][4];                                                 // this stage's and the next one's
        // Loads without a condition, so that they stay in flight until their stage is split: boards beyond the batch
        // repeat the last one (their outputs are dropped), terms beyond K repeat real ones (and are cleared below).
        const float* src_row[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) src_row[r] = L.in + (size_t)min(row0 + warp * 16 + r * 4 + sub, p.B - 1) * L.in_pitch;
        auto load = [&](int i, float4 (&x)[4]) {
            const int k = (kb0 + i) * kStageK + kv;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (VEC) x[r] = __ldcg(reinterpret_cast<const float4*>(src_row[r] + min(k, L.in_pitch - 4)));
                else x[r] = make_float4(__ldcg(src_row[r] + min(k, L.K - 1)), __ldcg(src_row[r] + min(k + 1, L.K - 1)),
                                        __ldcg(src_row[r] + min(k + 2, L.K - 1)), __ldcg(src_row[r] + min(k + 3, L.K - 1)));
            }
        };
        const int q = warp & 3, half = warp >> 2;                        // TMEM lane quadrant, 64 of the 128 outputs
        float group[64];
        bool flushed = false, ok = true;
        const int out_row = row0 + q * 32 + lane;
        float* const out = L.part + ((size_t)slice * p.B + out_row) * L.part_pitch + tile_n * kN + half * 64;
        const int out_n = L.part_pitch - (tile_n * kN + half * 64);      // outputs of this thread that exist
        // a group's sums -> the slice; further groups of a CTA that takes the whole layer are added to it in place
        auto flush = [&]() {
            if (out_row < p.B) {
#pragma unroll
                for (int j = 0; j < 64; j += 4) {
                    if (L.part_vec && j + 4 <= out_n) {
                        float4* at = reinterpret_cast<float4*>(out + j);
                        float4 v = make_float4(group[j], group[j + 1], group[j + 2], group[j + 3]);
                        if (flushed) {
                            const float4 o = *at;
                            v = make_float4(__fadd_rn(o.x, v.x), __fadd_rn(o.y, v.y), __fadd_rn(o.z, v.z), __fadd_rn(o.w, v.w));
                        }
                        *at = v;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (j + e < out_n) out[j + e] = flushed ? __fadd_rn(out[j + e], group[j + e]) : group[j + e];
                    }
                }
            }
            flushed = true;
        };
        auto drain = [&](int c) {                                        // chunk c of the layer
            const int acc = (c - chunk0) & 1;
            const bool good = mbar_wait(acc_full(acc), (uint32_t)((c - chunk0) >> 1) & 1u, abort_flag);
            if (!__all_sync(0xffffffffu, good)) { ok = false; return; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t t = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 2 * kN + half * 64);
            if (c == chunk0 || c % kHeadFcGroup == 0) {
#pragma unroll
                for (int j = 0; j < 64; ++j) group[j] = -0.0f;          // -0 + v is v for every v
            }
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                uint32_t r[8], small[8];
                tmem_ld8(t + h * 8, r);
                tmem_ld8(t + kN + h * 8, small);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float v = __fadd_rn(__uint_as_float(r[j]), fminf(__uint_as_float(small[j]), FLT_MAX));   // (NaN -> FLT_MAX)
                    group[h * 8 + j] = __fadd_rn(group[h * 8 + j], v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(acc));
            if (c % kHeadFcGroup == kHeadFcGroup - 1 || c + 1 == chunk1) flush();
        };
        load(0, xs[0]);
        load(1, xs[1]);
        int c_drained = chunk0;
        auto stage = [&](int i, float4 (&x)[4]) {
            const int s = i % kStages;
            const bool good = mbar_wait(empty(s), ((uint32_t)(i / kStages) & 1u) ^ 1u, abort_flag);
            if (!__all_sync(0xffffffffu, good)) { ok = false; return; }
            uint8_t* dst = smem + s * kStageBytes;
            // the layer's last block: terms beyond K have weights of zero, but an infinity repeated there would make NaN
            const int left = L.K - ((kb0 + i) * kStageK + kv);
            if (kb0 + i == L.k_blocks - 1 && left < 4) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (left < 1) x[r].x = 0.0f;
                    if (left < 2) x[r].y = 0.0f;
                    if (left < 3) x[r].z = 0.0f;
                    x[r].w = 0.0f;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int row = warp * 16 + r * 4 + sub;
                uint32_t h0, m0, l0, h1, m1, l1;
                split2(x[r].x, x[r].y, h0, m0, l0);
                split2(x[r].z, x[r].w, h1, m1, l1);
                // 64-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r / 2 % 4)
                uint8_t* at = dst + row * kRowBytes + (((kv >> 3) ^ ((row >> 1) & 3)) << 4) + (kv & 4) * 2;
                *reinterpret_cast<uint2*>(at) = make_uint2(h0, h1);
                *reinterpret_cast<uint2*>(at + kTileBytes) = make_uint2(m0, m1);
                *reinterpret_cast<uint2*>(at + 2 * kTileBytes) = make_uint2(l0, l1);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(in_full(s));
            load(i + 2, x);
            // the chunk before the one this stage belongs to: its MMAs are complete or nearly so
            if (c_drained < chunk0 + i / stages_per_chunk) drain(c_drained++);
        };
        for (int i = 0; ok && i < n_stages; i += 2) {
            stage(i, xs[0]);
            if (ok && i + 1 < n_stages) stage(i + 1, xs[1]);
        }
        while (ok && c_drained < chunk1) drain(c_drained++);
        if (!ok) { *abort_flag = 1; atomicExch(p.error, 3); }
    }

    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);    // copies in flight into shared memory land first
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
}

}  // namespace

size_t head_fc_packed_bytes(int K, int N) {
    return (size_t)((N + kN - 1) / kN) * ((K + kStageK - 1) / kStageK) * kOperandBytes;
}

// The three terms of a weight, as split2 makes them, but a finite one has finite terms up to fp32's largest number.
__device__ __forceinline__ void split_weight(float x, uint16_t (&t)[3]) {
    for (int s = 0; s < 3; ++s) {
        float lead = __bfloat162float(__float2bfloat16_rn(x));
        if (fabsf(lead) == INFINITY && fabsf(x) < INFINITY) lead = __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
        t[s] = (uint16_t)(__float_as_uint(lead) >> 16);
        x = __fsub_rn(x, lead);
    }
}
// w [N][K] fp32 -> blocks [output tile][32 inner terms][split term] of 128 outputs x 32 terms in bf16, 64 bytes an
// output, 16-byte chunks permuted by the 64-byte swizzle; outputs and terms beyond N and K are zero.
__global__ void head_fc_pack_kernel(const float* __restrict__ w, int K, int N, int k_blocks, uint8_t* __restrict__ packed) {
    const int tile = blockIdx.y, kb = blockIdx.x;
    uint8_t* block = packed + ((size_t)tile * k_blocks + kb) * kOperandBytes;
    for (int i = threadIdx.x; i < kN * kStageK / 2; i += blockDim.x) {
        const int r = i / (kStageK / 2), k = (i % (kStageK / 2)) * 2;
        const int n = tile * kN + r, gk = kb * kStageK + k;
        const float* src = w + (size_t)n * K + gk;
        uint16_t t0[3], t1[3];
        split_weight(n < N && gk < K ? src[0] : 0.0f, t0);
        split_weight(n < N && gk + 1 < K ? src[1] : 0.0f, t1);
        for (int s = 0; s < 3; ++s)
            *reinterpret_cast<uint32_t*>(block + s * kTileBytes + r * kRowBytes + (((k >> 3) ^ ((r >> 1) & 3)) << 4) + (k & 7) * 2) = t0[s] | (uint32_t)t1[s] << 16;
    }
}
int head_fc_pack(const float* w_dev, int K, int N, void* packed_dev, cudaStream_t st) {
    const int kb = (K + kStageK - 1) / kStageK;
    head_fc_pack_kernel<<<dim3(kb, (N + kN - 1) / kN), 256, 0, st>>>(w_dev, K, N, kb, static_cast<uint8_t*>(packed_dev));
    OB200_CUDA_OK(cudaGetLastError());
    return OB200_OK;
}

void head_fc_shape(HeadFcLayer* l, int K, int N) {
    l->K = K;
    l->n_tiles = (N + kN - 1) / kN;
    l->k_blocks = (K + kStageK - 1) / kStageK;
    // a short inner dimension (the 2 / 1-channel heads: 450 and 225 terms) in shorter chunks, so that there is something
    // to spread; a long one (7,200) in chunks of 256: 29 chunks x 4 output tiles fill the SMs with one row of tiles
    l->chunk_k = K <= 1024 ? 128 : 256;
    l->chunks = (K + l->chunk_k - 1) / l->chunk_k;
}

// Chunks per CTA for a batch: one, a group, or all.  The cheapest by the number of stages the busiest SM works off,
// plus eight for a CTA's fill and drain; with a few tiles of boards single chunks win, from some thousand boards on
// whole rows do (and write no partial sums but the result).
int head_fc_plan(HeadFcLayer* l, int n_layers, int B, int sms) {
    const long long m = (B + kM - 1) / kM;
    long long best_cost = 0;
    int best = -1;
    for (int mode = 0; mode < 3; ++mode) {
        long long ctas = 0, longest = 0;
        for (int i = 0; i < n_layers; ++i) {
            const int per = mode == 0 ? 1 : mode == 1 ? kHeadFcGroup : l[i].chunks;
            ctas += m * l[i].n_tiles * ((l[i].chunks + per - 1) / per);
            const long long st = (long long)(per < l[i].chunks ? per : l[i].chunks) * (l[i].chunk_k / kStageK) + 8;
            longest = st > longest ? st : longest;
        }
        const long long cost = (ctas + sms - 1) / sms * longest;
        if (best < 0 || cost <= best_cost) { best_cost = cost; best = mode; }
    }
    for (int i = 0; i < n_layers; ++i) {
        l[i].chunks_per_slice = best == 0 ? 1 : best == 1 ? kHeadFcGroup : l[i].chunks;
        l[i].slices = (l[i].chunks + l[i].chunks_per_slice - 1) / l[i].chunks_per_slice;
        l[i].slice_group = l[i].chunks_per_slice == 1 ? kHeadFcGroup : 1;
    }
    return best;
}

int launch_head_fc(const HeadFcLayer* layers, int n_layers, int B, cudaStream_t st) {
    if (n_layers < 1 || n_layers > 2 || B < 1) return set_error(OB200_ERR_INVALID, "head FC: bad arguments");
    int dev = 0;
    OB200_CUDA_OK(cudaGetDevice(&dev));
    static bool configured[64] = {false};
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        OB200_CUDA_OK(cudaFuncSetAttribute(head_fc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        OB200_CUDA_OK(cudaFuncSetAttribute(head_fc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    SplitParams p;
    p.B = B;
    p.error = device_error_word();
    if (!p.error) return set_error(OB200_ERR_CUDA, "head FC: cannot resolve the device error word");
    int entries = 0;
    bool vec = true;
    for (int i = 0; i < n_layers; ++i) {
        p.layer[i] = layers[i];
        vec = vec && (layers[i].in_pitch & 3) == 0 && ((uintptr_t)layers[i].in & 15) == 0;
        p.layer[i].part_vec = (layers[i].part_pitch & 3) == 0 && ((uintptr_t)layers[i].part & 15) == 0;
        entries += layers[i].n_tiles * layers[i].slices;
        if (i == 0) p.entries0 = entries;
    }
    if (n_layers == 1) p.layer[1] = p.layer[0];
    OB200_CUDA_OK(launch_dependent(vec ? head_fc_kernel<true> : head_fc_kernel<false>, dim3((B + kM - 1) / kM, entries), dim3(kThreads), (size_t)kSmemBytes, st, p));
    counters().launches.fetch_add(1, std::memory_order_relaxed);
    return OB200_OK;
}

}  // namespace ob200
