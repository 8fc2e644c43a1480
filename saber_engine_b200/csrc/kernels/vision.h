// Launch interface of the vision tower's kernels (vision.cu, vis_linear.cu).  Plain C types only.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace saber {

// Rows -> the GEMM's bf16 token operand: [K_total_pad/64][M_pad][128 bytes], 16-byte chunks XOR-swizzled
// by (row & 7).  Optional LayerNorm (weight and bias) on the way; optional row grouping (the merger's
// view [L/4, 4*K]): source row m lands in operand row m / group at column (m % group) * K.
struct VisRowsParams {
  const void* x;           // [M][ldx] fp32 (x_f32 = 1) or bf16
  int x_f32, ldx;
  const float* ln_w;       // [K] or null: no normalisation, a cast
  const float* ln_b;       // [K]
  float eps;
  uint8_t* tiled;
  int M, K;                // K a multiple of 8
  int K_pad;               // operand columns per SOURCE row, a multiple of 64 when group == 1 (zero filled past K)
  int M_pad;               // operand rows (>= ceil(M / group), a multiple of the GEMM's token tile)
  int group;               // 1 or 4 (K a multiple of 64 when > 1)
};

// x[m][:] += sum_i table[idx[m][i]][:] * wt[m][i]   (bilinear gather of the learned position table);
// weights and products rounded to bf16, the four products added left to right in bf16.
struct VisPosAddParams {
  __nv_bfloat16* x; int ldx;
  const __nv_bfloat16* table; int ldt;
  const int* idx;          // [M][4]
  const float* wt;         // [M][4]
  int M, K;
};

// Non-causal attention inside each image; head dim 72.  q, k and v: scratch of the sizes that saber_vis_attn_scratch gives.
struct VisAttnParams {
  const __nv_bfloat16* qkv; int ldq;     // [L][3 * width]: q | k | v, head-major inside each
  const float* cos_t; const float* sin_t; // [L][36]
  uint8_t* out_tiled; int M_pad;          // the projection GEMM's token operand (width columns)
  const int4* blocks;                     // 64 rows of an image each {first row of the image, rows of the image, first row (relative), 0}
  int heads, width;
  float scale;                            // 1 / sqrt(72)
  __nv_bfloat16* q; uint8_t* k; uint8_t* v;
  const int32_t* cu_rows;                 // [images + 1]
  const int32_t* kv_len;                  // [images]: rows of an image
  const int32_t* pages;                   // [images][max_pages]: the blocks of an image
  int images, max_pages, max_rows;
  uint32_t* err;
};

// out = epi(bf16(x W^T + bias)): epi 1 gelu (by tanh), 2 gelu (by the error function), 3 + res; bf16 rows (vis_linear.cu).
struct VisLinearParams {
  const uint8_t* w;        // [N_pad / 256][k-block of 64][256 rows of 128 bytes]
  const uint8_t* a;        // [k-block][M_pad][128 bytes]
  const float* bias;       // [N] or null
  const __nv_bfloat16* res; // epi 3: out's row stride, may alias out
  __nv_bfloat16* out;      // [M][ldo]
  float* ws;               // an SM: 128 x 256 floats
  uint32_t* counters;      // an SM: a word, zero between launches
  uint32_t* err;
  int M, M_pad, N, N_pad, K, ldo, epi;
};

}  // namespace saber

extern "C" int saber_vis_linear_launch(const saber::VisLinearParams* p, cudaStream_t stream);
extern "C" int saber_vis_rows_launch(const saber::VisRowsParams* p, cudaStream_t stream);
extern "C" int saber_vis_pos_add_launch(const saber::VisPosAddParams* p, cudaStream_t stream);
extern "C" int saber_vis_attn_launch(const saber::VisAttnParams* p, int n_blocks, cudaStream_t stream);
extern "C" int saber_vis_attn_scratch(int n_blocks, int rows, int heads, size_t* q, size_t* k, size_t* v);
