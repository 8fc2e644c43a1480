// The vision tower's own kernels: rows -> bf16 GEMM operand (cast or LayerNorm, optional 4-row
// grouping for the merger), the position-table gather, and non-causal attention with 2-D rotary
// embedding.  The tower's linears (patch embed, qkv, proj, fc1 + GELU, fc2 + residual, merger) run on
// vis_linear.cu with bias / activation / residual in the epilogue.
//
// Parity: the reference tower's op list and rounding points (crates/saber-kernels/hip/vision.hip:1-30):
// every linear rounds to bf16 once and the activation / residual work on the rounded value;
// LayerNorm, softmax and rotary arithmetic run in fp32; rotated q and k are rounded to bf16; the
// attention products run on tcgen05 (bf16 operands, fp32 accumulators).
#include "vision.h"
#include "flash_tc.h"
#include "launch.cuh"

namespace saber {

constexpr int kVisThreads = 128;
constexpr int kPrepThreads = 192;
constexpr int kVisMaxChunks = 5;     // 8-value chunks per thread: rows of up to 5120 values

// kLanes 32: a row per warp, four a CTA; 128: a row per CTA.
template <int kLanes>
__device__ __forceinline__ float row_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (kLanes == 32) return v;
  const int w = threadIdx.x >> 5;
  __syncthreads();                       // red may still be read from the previous call
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  return red[0] + red[1] + red[2] + red[3];
}

// Bound by memory (3 us for 4096 rows of 1152 at the copy rate).  A row per warp wherever it holds one: a row per CTA left most of the 128 threads
// without a second chunk and met at four barriers, and a condition beside every element's norm weight was a branch an element
// (15.4 us a launch; a 64 x 64 image has 84 of them and takes 9.1 ms, 9.7 before).
template <int kLanes, bool kF32>
__global__ void __launch_bounds__(kVisThreads) vis_rows_kernel(const VisRowsParams p) {
  __shared__ float red[4];
  pdl_trigger();
  pdl_wait();
  const int t = threadIdx.x & (kLanes - 1), m = blockIdx.x * (kVisThreads / kLanes) + threadIdx.x / kLanes;
  if (m >= p.M) return;
  const int nch = p.K_pad >> 3, live = p.K >> 3;
  float v[kVisMaxChunks][8];
#pragma unroll
  for (int i = 0; i < kVisMaxChunks; ++i) {
    const int c = t + i * kLanes;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    if (c < live) {
      if constexpr (kF32) {
        const float4* s = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + static_cast<size_t>(m) * p.ldx + c * 8);
        const float4 a = s[0], b = s[1];
        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
        v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
      } else {
        const uint4 raw = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.x) + static_cast<size_t>(m) * p.ldx + c * 8);
        const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(b[j]);
      }
    }
  }
  if (p.ln_w != nullptr) {
    float sum = 0.f, sq = 0.f;
#pragma unroll
    for (int i = 0; i < kVisMaxChunks; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += v[i][j];                    // (chunks past the row are zeros)
    const float mean = row_sum<kLanes>(sum, red) / static_cast<float>(p.K);
#pragma unroll
    for (int i = 0; i < kVisMaxChunks; ++i)
      if (t + i * kLanes < live) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float d = v[i][j] - mean; sq += d * d; }
      }
    const float rstd = rsqrtf(row_sum<kLanes>(sq, red) / static_cast<float>(p.K) + p.eps);
#pragma unroll
    for (int i = 0; i < kVisMaxChunks; ++i) {
      const int c = t + i * kLanes;
      if (c < live) {
        const float4* w4 = reinterpret_cast<const float4*>(p.ln_w + c * 8);
        const float4* b4 = reinterpret_cast<const float4*>(p.ln_b + c * 8);
        const float4 w0 = w4[0], w1 = w4[1], b0 = b4[0], b1 = b4[1];
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w}, b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = (v[i][j] - mean) * rstd * w[j] + b[j];
      }
    }
  }
  const int row_o = m / p.group;
  const int col_base = (m % p.group) * p.K;
#pragma unroll
  for (int i = 0; i < kVisMaxChunks; ++i) {
    const int c = t + i * kLanes;
    if (c >= nch) break;
    uint4 o;
    __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) ob[j] = __float2bfloat16(v[i][j]);   // (zeros up to the operand's end)
    const int col0 = col_base + c * 8;
    const int kb = col0 >> 6, chunk = (col0 & 63) >> 3;
    *reinterpret_cast<uint4*>(p.tiled + (static_cast<size_t>(kb) * p.M_pad + row_o) * 128 +
                              ((chunk ^ (row_o & 7)) << 4)) = o;
  }
}

__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16(x)); }

__global__ void __launch_bounds__(kVisThreads) vis_pos_add_kernel(const VisPosAddParams p) {
  pdl_wait();
  const int m = blockIdx.x;
  int id[4];
  float w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { id[i] = p.idx[m * 4 + i]; w[i] = rbf(p.wt[m * 4 + i]); }
  for (int k = threadIdx.x; k < p.K; k += kVisThreads) {
    float s = rbf(__bfloat162float(p.table[static_cast<size_t>(id[0]) * p.ldt + k]) * w[0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) s = rbf(s + rbf(__bfloat162float(p.table[static_cast<size_t>(id[i]) * p.ldt + k]) * w[i]));
    __nv_bfloat16* x = p.x + static_cast<size_t>(m) * p.ldx + k;
    *x = __float2bfloat16(__bfloat162float(*x) + s);
  }
}

// ------------------------------------------------------------------------------------ attention
// Non-causal attention inside each image, two launches: this one and the prompt attention of flash_tc.cu with every key visible.
// A CTA takes 64 rows of one image and one head: q and k turned (out[d] = x[d] cos - x[d+36] sin, out[d+36] = x[d+36] cos + x[d] sin,
// fp32, one rounding to bf16), q as rows of kVisDK values, k and the transposed v as the page of 64 keys that attention multiplies
// in place.  Bound by memory: 7 KB in and 7 KB out per row, 11 us at 4096 rows (14 us for the rotation in place before, which left keys and
// values in rows); all of a thread's loads are requested together.  With the attention behind it 147 us at 4096 rows (316 before) and 19 at 308
// (13: three key blocks one behind the other in 32 CTAs are a longer chain than the 80 CTAs of `mma.sync` had).
constexpr int kHd = 72, kHalf = 36;
constexpr int kVisDK = 80, kVisKeyTiles = 2, kVisVP = 96;          // the head in whole steps of the tensor cores; values up to 32 columns

__device__ __forceinline__ float4 bf4(const uint2 v) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ uint2 bf4(float a, float b, float c, float d) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

// The rotated halves of four values of each half of a head row.
__device__ __forceinline__ void rope4(const uint2 x1, const uint2 x2, const float4 c, const float4 s, uint2& lo, uint2& hi) {
  const float4 a = bf4(x1), b = bf4(x2);
  lo = bf4(a.x * c.x - b.x * s.x, a.y * c.y - b.y * s.y, a.z * c.z - b.z * s.z, a.w * c.w - b.w * s.w);
  hi = bf4(b.x * c.x + a.x * s.x, b.y * c.y + a.y * s.y, b.z * c.z + a.z * s.z, b.w * c.w + a.w * s.w);
}

__global__ void __launch_bounds__(kPrepThreads) vis_prep_kernel(const VisAttnParams p) {
  constexpr int kPer = 64 * 9 / kPrepThreads;
  static_assert(kPer * kPrepThreads == 64 * 9 && kHalf == 36, "nine four-value groups of a half row, nine pieces of a row");
  __shared__ __align__(16) uint8_t v_s[64 * kHd * 2 + 8 * 16];
  pdl_wait();
  const int4 blk = p.blocks[blockIdx.x];
  const int h = blockIdx.y, m0 = blk.x + blk.z, n = min(64, blk.y - blk.z);
  uint8_t* kp = p.k + (static_cast<size_t>(blockIdx.x) * p.heads + h) * kVisKeyTiles * 8192;
  uint8_t* vp = p.v + (static_cast<size_t>(blockIdx.x) * p.heads + h) * kVisVP * 128;
  uint2 q1[kPer], q2[kPer], k1[kPer], k2[kPer];
  uint4 v[kPer];
  float4 cs[kPer], sn[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = threadIdx.x + i * kPrepThreads, r = e / 9, g = e - r * 9;
    q1[i] = q2[i] = k1[i] = k2[i] = make_uint2(0u, 0u);            // (keys past the image: zeros, their probabilities are)
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    cs[i] = sn[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) {
      const __nv_bfloat16* row = p.qkv + static_cast<size_t>(m0 + r) * p.ldq + h * kHd;
      q1[i] = *reinterpret_cast<const uint2*>(row + g * 4);
      q2[i] = *reinterpret_cast<const uint2*>(row + kHalf + g * 4);
      k1[i] = *reinterpret_cast<const uint2*>(row + p.width + g * 4);
      k2[i] = *reinterpret_cast<const uint2*>(row + p.width + kHalf + g * 4);
      v[i] = *reinterpret_cast<const uint4*>(row + 2 * p.width + g * 8);
      cs[i] = *reinterpret_cast<const float4*>(p.cos_t + static_cast<size_t>(m0 + r) * kHalf + g * 4);
      sn[i] = *reinterpret_cast<const float4*>(p.sin_t + static_cast<size_t>(m0 + r) * kHalf + g * 4);
    }
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = threadIdx.x + i * kPrepThreads, r = e / 9, g = e - r * 9;
    *reinterpret_cast<uint4*>(v_s + r * (kHd * 2) + (r >> 3) * 16 + g * 16) = v[i];
    auto key = [&](int col) { return kp + (col >> 6) * 8192 + r * 128 + ((((col >> 3) & 7) ^ (r & 7)) << 4) + (col & 7) * 2; };
    uint2 lo, hi;
    rope4(k1[i], k2[i], cs[i], sn[i], lo, hi);
    *reinterpret_cast<uint2*>(key(g * 4)) = lo;
    *reinterpret_cast<uint2*>(key(kHalf + g * 4)) = hi;
    if (g == 8) *reinterpret_cast<uint4*>(key(kHd)) = make_uint4(0u, 0u, 0u, 0u);
    if (r < n) {
      __nv_bfloat16* q = p.q + (static_cast<size_t>(m0 + r) * p.heads + h) * kVisDK;
      rope4(q1[i], q2[i], cs[i], sn[i], lo, hi);
      *reinterpret_cast<uint2*>(q + g * 4) = lo;
      *reinterpret_cast<uint2*>(q + kHalf + g * 4) = hi;
      if (g == 8) *reinterpret_cast<uint4*>(q + kHd) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 8 * kHd / 2; e += kPrepThreads) {  // eight keys of two value columns (columns past the head are never read)
    const int d = (e >> 3) * 2, c = e & 7;                         // the rows' pad of 16 bytes per eight puts the 32 lanes' words on 32 banks
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const uint32_t*>(v_s + (c * 8 + j) * (kHd * 2) + c * 16 + d * 2);
    uint4 o;
    o.x = __byte_perm(w[0], w[1], 0x5410); o.y = __byte_perm(w[2], w[3], 0x5410); o.z = __byte_perm(w[4], w[5], 0x5410); o.w = __byte_perm(w[6], w[7], 0x5410);
    *reinterpret_cast<uint4*>(vp + d * 128 + ((c ^ (d & 7)) << 4)) = o;
    o.x = __byte_perm(w[0], w[1], 0x7632); o.y = __byte_perm(w[2], w[3], 0x7632); o.z = __byte_perm(w[4], w[5], 0x7632); o.w = __byte_perm(w[6], w[7], 0x7632);
    *reinterpret_cast<uint4*>(vp + (d + 1) * 128 + ((c ^ ((d + 1) & 7)) << 4)) = o;
  }
}

}  // namespace saber

extern "C" int saber_vis_rows_launch(const saber::VisRowsParams* p, cudaStream_t stream) {
  using namespace saber;
  if (p->M <= 0) return 0;
  if ((p->K & 7) || (p->K_pad & 7) || p->K_pad < p->K || p->K_pad > kVisMaxChunks * kVisThreads * 8 ||
      (p->group != 1 && p->group != 4) || (p->group == 1 && (p->K_pad & 63)) ||
      (p->group > 1 && ((p->K & 63) || p->K_pad != p->K)) || (p->ldx & 7) || (p->M + p->group - 1) / p->group > p->M_pad)
    return static_cast<int>(cudaErrorInvalidValue);
  const dim3 warps((p->M + 3) / 4), ctas(p->M), threads(kVisThreads);
  if (p->K_pad <= kVisMaxChunks * 32 * 8)
    return static_cast<int>(p->x_f32 ? launch(vis_rows_kernel<32, true>, warps, threads, 0, stream, 0, *p) : launch(vis_rows_kernel<32, false>, warps, threads, 0, stream, 0, *p));
  return static_cast<int>(p->x_f32 ? launch(vis_rows_kernel<128, true>, ctas, threads, 0, stream, 0, *p) : launch(vis_rows_kernel<128, false>, ctas, threads, 0, stream, 0, *p));
}

extern "C" int saber_vis_pos_add_launch(const saber::VisPosAddParams* p, cudaStream_t stream) {
  using namespace saber;
  if (p->M <= 0) return 0;
  return static_cast<int>(saber::launch(vis_pos_add_kernel, dim3(p->M), dim3(kVisThreads), 0, stream, 0, *p));
}

extern "C" int saber_vis_attn_launch(const saber::VisAttnParams* p, int n_blocks, cudaStream_t stream) {
  using namespace saber;
  if (n_blocks <= 0) return 0;
  if ((p->width & 7) || p->heads * kHd != p->width || (p->ldq & 7) || p->images <= 0 || p->max_rows <= 0) return static_cast<int>(cudaErrorInvalidValue);
  const cudaError_t e = launch(vis_prep_kernel, dim3(n_blocks, p->heads), dim3(kPrepThreads), 0, stream, 0, *p);
  if (e != cudaSuccess) return static_cast<int>(e);
  FlashParams f = {};
  f.q = p->q;
  f.k = p->k;
  f.v = p->v;
  f.k_stride = static_cast<size_t>(kVisKeyTiles) * 8192;
  f.v_stride = static_cast<size_t>(kVisVP) * 128;
  f.cu_rows = p->cu_rows;
  f.kv_len = p->kv_len;
  f.block_table = p->pages;
  f.out.p = p->out_tiled;
  f.out.M_pad = p->M_pad;
  f.nseq = p->images;
  f.H = f.G = p->heads;
  f.DK = kVisDK;
  f.V = kHd;
  f.VP = kVisVP;
  f.n_blocks = n_blocks;
  f.max_blocks = p->max_pages;
  f.max_rows = p->max_rows;
  f.full = 1;
  f.out_scale = 1.f;
  f.scale = p->scale;
  f.err = p->err;
  return saber_flash_tc(&f, stream);
}

extern "C" int saber_vis_attn_scratch(int n_blocks, int rows, int heads, size_t* q, size_t* k, size_t* v) {
  using namespace saber;
  *q = static_cast<size_t>(rows) * heads * kVisDK * 2;
  *k = static_cast<size_t>(n_blocks) * heads * kVisKeyTiles * 8192;
  *v = static_cast<size_t>(n_blocks) * heads * kVisVP * 128;
  return 0;
}
