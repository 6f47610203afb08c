// Launchers shared between the translation units of the library (C++ linkage).
#pragma once
#include "common.h"

namespace ob200 {

int launch_encode_gomoku(const int16_t* history, const uint8_t* n_hist, const uint8_t* to_move, int32_t B,
                         int32_t board_size, int32_t planes, int32_t out_channels, void* board_tensor_out,
                         cudaStream_t stream, int dtype = 0);
int launch_encode_go(const int8_t* stones, const int32_t* ko_point, const uint8_t* to_move, const uint32_t* legal_bits,
                     int32_t B, int32_t board_size, int32_t out_channels, void* board_tensor_out, cudaStream_t stream,
                     int dtype = 0);
int launch_encode_gomoku3(const int8_t* stones, const uint8_t* to_move, int32_t B, int32_t board_size, int32_t out_channels,
                          void* board_tensor_out, cudaStream_t stream, int dtype = 0);
int launch_encode_chess(const int8_t* pieces, const int32_t* meta, const uint32_t* legal_to, int32_t B,
                        int32_t out_channels, void* board_tensor_out, cudaStream_t stream, int dtype = 0);
int launch_planes_to_board_tensor(const float* planes_nchw, int32_t B, int32_t C, int32_t board_size,
                                  int32_t out_channels, void* board_tensor_out, cudaStream_t stream, int dtype = 0);
// Opaque storage of a CUtensorMap (128 bytes, 64-byte aligned) so that only the convolution's
// translation unit needs the driver API header.
struct alignas(64) BoardTensorMap { unsigned char opaque[128]; };
int make_board_tensor_map(const void* base, long long rows, int box_rows, BoardTensorMap* out, int channels = 64);
int conv_halo_rows(int S);   // 64-channel kernel: load boxes have 128 + 2 * conv_halo_rows(S) rows
// res_map: the residual tensor through a 128-row-box map (a store map of that buffer), or null
int launch_conv3x3_maps(const BoardTensorMap& in_map, const BoardTensorMap& out_map, const BoardTensorMap* res_map,
                        const void* packed_w, const float* bias, int B, int S, int relu, cudaStream_t st, int dtype = 0);
int* device_error_word();
// The whole 64-filter tower as one cooperative launch (tower_fused.cu).
size_t tower_fused_layer_bytes();
void tower_fused_fill_layer(void* dst, const BoardTensorMap* in_map, const BoardTensorMap& out_map,
                            const BoardTensorMap* res_map, const void* w, const float* bias);
size_t tower_fused_smem_bytes(int S, int n_layers);   // 0: does not fit
int launch_conv_tower(const BoardTensorMap& stem_in_map, const void* layers_dev, int n_layers, int* flags, int tiles_pitch,
                      int* done, int epoch, int B, int S, cudaStream_t st, int dtype = 0);
// The 64-filter tower with the boards resident in shared memory (tower_resident.cu): boards up to
// 15x15, one ordinary launch.
// The even and the odd columns of a 64-channel board tensor of B boards as 4-D maps (channel, pair of cells, row, board);
// a box is one board's plane, (S + 2) / 2 pairs x (S + 1) rows, what lies outside the grid reads as zero.
struct BoardPlaneMaps { BoardTensorMap even, odd; };
int make_board_plane_maps(const void* base, int S, int B, BoardPlaneMaps* out);
// The heads' 1x1 convolutions (head_conv.cuh).  w: blocks [group of up to 64 channels][64-channel K slice][split term]
// of (channels of the group rounded up to 16) rows x 128 bytes, 128-byte swizzle; scale, bias: [hc].
struct HeadConvWeights { const uint8_t* w; const float *scale, *bias; int hc, pc; };
size_t head_conv_packed_bytes(int hc, int C);
void head_conv_pack(const float* w, int hc, int C, int dtype, void* packed_out, float* scale_out);   // w [hc][C], host
bool tower_resident_covers(int S, int n_layers);
int tower_resident_head_channels_max();
// head (optional): the heads' 1x1 convolutions come along as one more layer (results as launch_head_conv's).
// enc_hist != null: the input is not read through `in` but written by the kernel from Gomoku move histories
// ([B][16] int16, 16-byte aligned; history lengths and sides to move [B]; 17 or 19 planes), as launch_encode_gomoku would.
int launch_conv_tower_resident(const BoardPlaneMaps& in, const BoardPlaneMaps& out, const void* const* layers_dev, const float* bias,
                               int n_layers, int B, int S, cudaStream_t st, const HeadConvWeights* head = nullptr, float* hp = nullptr, float* hv = nullptr,
                               int hp_pitch = 0, int hv_pitch = 0, int dtype = 0, const int16_t* enc_hist = nullptr,
                               const uint8_t* enc_nh = nullptr, const uint8_t* enc_tm = nullptr, int enc_planes = 0);
// Towers of 128 / 256 channels (tower_wide.cu): cin a multiple of 64 up to 256, cout 128 or 256,
// taps 9 (3x3) or 1 (1x1).  in_map: boxes of conv_wide_box_rows() rows over a cin-channel tensor;
// out_map / res_map (residual, or null): boxes of 128 rows over a cout-channel tensor.
// out_f32 (optional): fp32 [positions][cout] output by plain stores instead of the bf16 tensor.
bool conv_wide_covers(int cin, int cout);
int conv_wide_box_rows();
size_t conv_wide_packed_bytes(int cin, int cout, int taps);
int conv_wide_pack(const float* w, const float* scale, int cout, int cin_real, int cin, int taps, void* packed_out, int dtype = 0);
int launch_conv_wide_maps(const BoardTensorMap& in_map, const BoardTensorMap& out_map, const BoardTensorMap* res_map,
                          const void* packed_w, const float* bias, int B, int S, int cin, int cout, int taps, int relu,
                          cudaStream_t st, float* out_f32 = nullptr, int dtype = 0);
// The same layers on 8x8 boards over the cells alone (tower_board8.cu).  A tensor of B boards as 4-D maps (channel, x, y,
// board); a box is 64 channels of one board row of 2 (m[0]) or 4 (m[1]) boards, what lies outside the boards reads as
// zero.  Padding positions of the output are left as they are (zero in a handle's tensors).
struct BoardRowMaps { BoardTensorMap m[2]; };
int make_board_row_maps(const void* base, int S, int B, int channels, BoardRowMaps* out);
bool conv_board8_covers(int S, int cin, int cout);
void conv_board8_pack(const float* w, const float* scale, int cout, int cin_real, int cin, void* packed_out, int dtype);
int launch_conv_board8(const BoardRowMaps& in, const BoardRowMaps& out, const BoardRowMaps* res, const void* packed_w, const float* bias,
                       int B, int cin, int cout, int relu, cudaStream_t st, int dtype);

// C: channels of the tower board tensor (a multiple of 64).
// hp [B][hp_pitch], hv [B][hv_pitch]: a board's policy / value head channels, flattened as c * S*S + y * S + x
int launch_head_conv(const void* tower, const HeadConvWeights& head, float* hp, float* hv, int hp_pitch, int hv_pitch, int B, int S,
                     cudaStream_t st, int C = 64, int dtype = 0);
// A fully connected layer of a head on the tensor cores in fp32 precision (head_fc.cu): its sums leave as `slices`
// partial results [slice][B][part_pitch], to be added in order - in runs of slice_group first, when that is above 1.
constexpr int kHeadFcGroup = 3;
struct HeadFcLayer {
    const float* in;          // [B][in_pitch]
    int in_pitch, K;
    const uint8_t* w;         // head_fc_pack
    int n_tiles, k_blocks, chunk_k, chunks, chunks_per_slice, slices, slice_group;
    float* part;
    int part_pitch;           // outputs beyond it are dropped
    int part_vec;             // set by the launcher: rows may be written 16 bytes at a time
};
size_t head_fc_packed_bytes(int K, int N);
int head_fc_pack(const float* w_dev, int K, int N, void* packed_dev, cudaStream_t st);   // w [N][K] on the device
void head_fc_shape(HeadFcLayer* l, int K, int N);
int head_fc_plan(HeadFcLayer* l, int n_layers, int B, int sms);
int launch_head_fc(const HeadFcLayer* layers, int n_layers, int B, cudaStream_t st);
// What is left of both heads in one launch: partial sums + bias -> logits (or softmax of them), partial sums + bias ->
// ReLU -> value FC2 -> tanh.  policy.part may be null: the logits are in policy_out already (convolution planes).
// error_out (optional): receives the device error word as the kernels ahead have left it.
int launch_head_tails(const HeadFcLayer& policy, const float* bp, float* policy_out, int policy_size, int softmax,
                      const HeadFcLayer& value, const float* b1, int H, const float* w2, float b2, float* value_out, int B,
                      cudaStream_t st, int* error_out = nullptr);
// value_layer: the value head's first FC (its in / part fields are filled in here)
int launch_value_head_static(const void* tower, const HeadConvWeights& value_conv, const HeadFcLayer& value_layer,
                             const float* b1, const float* w2, float b2, int H, int B, int S, float* value_out,
                             cudaStream_t st, int dtype = 0);
size_t value_head_static_capacity();

}  // namespace ob200
