// Chunks of sixteen tokens on the tensor cores with fp32 factors: what the prompt scans of delta_chunk.cu and cdelta_chunk.cu share.
//
// An fp32 factor enters `mma.sync` as a sum of three bf16 values (24 bits, the fp32 mantissa); of the nine products of two such sums the six whose
// sizes matter are added, the small ones first, with fp32 accumulation.
#pragma once
#include "mla_device.cuh"
#include "ptx_sm100.cuh"

namespace saber {

constexpr int kDcTok = 16, kDcCols = 32, kDcStages = 3;
constexpr int kDcThreads = 160;                     // four warps of a scan, one that keeps the copies going
constexpr int kDcVRow = kDcCols + 4;                // floats of a value row (lanes of a fragment hit all banks)
constexpr int kDcV = kDcTok * kDcVRow * 4;
constexpr int kDcPairRow = 48;                      // bytes of a row of a 16 x 16 matrix (eight rows hit all banks)
constexpr int kDcMat = 3 * 16 * kDcPairRow;         // three parts

// Chunks of sequence j occupy the slots from (first row / 16) + j on.
__device__ __forceinline__ int dc_slot(int r0, int j) { return r0 / kDcTok + j; }
// byte of channel c of a token inside one part of k or q
__device__ __forceinline__ int dc_at(int tok, int c) { return (c >> 6) * kDcTok * 128 + tok * 128 + (((((c & 63) >> 3) ^ tok) & 7) << 4) + (c & 7) * 2; }

// Two fp32 values as three bf16 pairs whose sums they are (to 24 bits).
__device__ __forceinline__ void dc_split(float a, float b, uint32_t& s0, uint32_t& s1, uint32_t& s2) {
  s0 = pack2(a, b);
  a -= __uint_as_float(s0 << 16);
  b -= __uint_as_float(s0 & 0xffff0000u);
  s1 = pack2(a, b);
  a -= __uint_as_float(s1 << 16);
  b -= __uint_as_float(s1 & 0xffff0000u);
  s2 = pack2(a, b);
}

// element (i, j) of a 16 x 16 matrix in three parts
__device__ __forceinline__ void dc_store_part3(uint8_t* mat, int i, int j, float v) {
  __nv_bfloat16 b = __float2bfloat16(v);
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    *reinterpret_cast<__nv_bfloat16*>(mat + e * 16 * kDcPairRow + i * kDcPairRow + j * 2) = b;
    v -= __bfloat162float(b);
    b = __float2bfloat16(v);
  }
}

// A (three parts) times B (three parts) onto c: the products whose parts' sizes matter, small ones first
template <int kN>
__device__ __forceinline__ void dc_mma6(float (&c)[kN][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * kN]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    constexpr int ea[6] = {0, 1, 2, 0, 1, 0}, eb[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
    for (int n = 0; n < kN; ++n) mma16816(c[n], a[ea[e]], b[eb[e]][2 * n], b[eb[e]][2 * n + 1]);
  }
}

// The same over many steps: the large products in a sum of their own (the tensor cores cut a sum's last place off, once a product: small ones
// added to a large sum would cost as much as the large ones).  Two sums in turn: four products between two on the same accumulator.
template <int kN>
__device__ __forceinline__ void dc_mma6_apart(float (&c)[kN][4], float (&lo)[kN][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * kN]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    constexpr int ea[6] = {0, 1, 2, 0, 1, 0}, eb[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
    for (int n = 0; n < kN; ++n) mma16816(e < 5 ? lo[n] : c[n], a[ea[e]], b[eb[e]][2 * n], b[eb[e]][2 * n + 1]);
  }
}
template <int kN>
__device__ __forceinline__ void dc_mma6_apart(float (&c)[2][kN][4], float (&d)[2][kN][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * kN], const uint32_t (&g)[3][2 * kN]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    constexpr int ea[6] = {0, 1, 2, 0, 1, 0}, eb[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
    for (int n = 0; n < kN; ++n) mma16816(c[e < 5][n], a[ea[e]], b[eb[e]][2 * n], b[eb[e]][2 * n + 1]);
#pragma unroll
    for (int n = 0; n < kN; ++n) mma16816(d[e < 5][n], a[ea[e]], g[eb[e]][2 * n], g[eb[e]][2 * n + 1]);
  }
}

// Two products of one step each, in turn.
template <int kN, int kM>
__device__ __forceinline__ void dc_mma6(float (&c)[kN][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * kN], float (&d)[kM][4], const uint32_t (&f)[3][4],
                                        const uint32_t (&g)[3][2 * kM]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    constexpr int ea[6] = {0, 1, 2, 0, 1, 0}, eb[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
    for (int n = 0; n < kN; ++n) mma16816(c[n], a[ea[e]], b[eb[e]][2 * n], b[eb[e]][2 * n + 1]);
#pragma unroll
    for (int n = 0; n < kM; ++n) mma16816(d[n], f[ea[e]], g[eb[e]][2 * n], g[eb[e]][2 * n + 1]);
  }
}

// A product of many factors as the sum of two fp32 numbers: sixteen roundings would show in the results.
struct DcProduct {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float g) {
    const float p = __fmul_rn(hi, g);
    lo = fmaf(lo, g, fmaf(hi, g, -p));
    hi = p;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
};

// the fragment of two accumulator tiles (rows x 16 columns) as an operand in three parts
__device__ __forceinline__ void dc_operand(const float (&x)[4], const float (&y)[4], uint32_t (&a)[3][4]) {
  dc_split(x[0], x[1], a[0][0], a[1][0], a[2][0]);
  dc_split(x[2], x[3], a[0][1], a[1][1], a[2][1]);
  dc_split(y[0], y[1], a[0][2], a[1][2], a[2][2]);
  dc_split(y[2], y[3], a[0][3], a[1][3], a[2][3]);
}

template <typename Kernel>
static int dc_allow(Kernel kernel, bool (&ready)[64], int smem) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return static_cast<int>(cudaErrorInvalidDevice);
  if (ready[dev]) return 0;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  ready[dev] = e == cudaSuccess;
  return static_cast<int>(e);
}

}  // namespace saber
