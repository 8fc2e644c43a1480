// Gated delta rule over prompt portions on the tensor cores: sixteen tokens at a time, the state in registers.
//
// With G_i = g_1 .. g_i and D_ij = g_{j+1} .. g_i (products, no quotients), the rule of delta.h over a chunk of sixteen tokens is
//     u = T (beta (v - G S_0^T k)),   T = (1 + A)^-1,   A_ij = beta_i D_ij (k_j . k_i) for j < i
//     o_i = G_i S_0^T q_i + sum_{j<=i} D_ij (k_j . q_i) u_j
//     S = G_16 S_0 + sum_j k_j (D_16j u_j)^T
// Everything that meets the state is a product of 16 columns of it with 16 keys or queries, in three bf16 parts each (chunk16.cuh).  The state is an
// fp32 accumulator that is only ever scaled and added to in fp32: S = G_16 S + (products).
//
//   prep   a CTA per (chunk, key head): convolution, silu, unit norms, the chunk's dot products; per value head the decays, T by forward
//          substitution and the pair weights
//   scan   a CTA per (sequence, head, 32 value columns): two pairs of warps, sixteen columns a pair, half of the keys a warp.  Accumulator
//          fragments of S^T are the operand fragments of the next product, and those of S^T K^T are (scaled) the operand of T.  The halves of
//          a product meet in shared memory.  Records of the next chunks arrive by bulk copies.
// Bound by the chain of four dependent products a chunk: 1.27 us of it, 128 chunks one behind the other.  2048 tokens, 32 heads of 128 x 128: scan 162 us
// (512 blocks of four tokens, fp32 multiply-adds: 441), preparation 95 (58).  A quarter of the keys a warp (eight warps) took 203: a third meeting costs
// more than the shorter sums save.  Error against 64 bits over 37 to 2048 tokens and weak to strong decays: 1.4 to 2.2e-7 of the output and 1.3 to 3.6e-7
// of the state, the four-token scan's 1.3 to 2.2e-7 and 1.4 to 3.9e-7 (large products in sums of their own, decays as pairs of fp32 numbers, and X added
// to the product with T's part below the diagonal are what that takes).
#include "chunk16.cuh"
#include "delta.h"
#include "launch.cuh"
#include "scan_records.cuh"

namespace saber {

constexpr int kDcSmall = 2 * kDcMat + 4 * kDcTok * 4;      // T | pair weights | beta | beta G | G | D_16j
__host__ __device__ constexpr int dc_kq(int DP) { return 6 * kDcTok * DP * 2; }          // k parts | q parts, each [part][64 channels][token][128 bytes]

struct DcLayout {                                   // of a chunk's slot, in bytes: [HK] k | q, [H][slices] v, [H] small
  size_t v, small, bytes;
};
__host__ __device__ inline DcLayout dc_layout(int H, int HK, int DP, int VP) {
  const size_t slices = static_cast<size_t>((VP + kDcCols - 1) / kDcCols);
  DcLayout l;
  l.v = static_cast<size_t>(HK) * dc_kq(DP);
  l.small = l.v + H * slices * kDcV;
  l.bytes = (l.small + static_cast<size_t>(H) * kDcSmall + 127) / 128 * 128;
  return l;
}
__device__ __forceinline__ int dc_state_slot(const DeltaParams& p, int j) {
  const int s = p.slots[j];
  if (s >= p.n_slots) {
    if (p.err) atomicCAS(p.err, 0u, static_cast<uint32_t>(kErrBadIndex));
    return -1;
  }
  return s;
}

// convolution + silu of channel c (column col of the rows) for up to sixteen rows from m on (row t of its sequence, at position pos)
template <int TAPS>
__device__ __forceinline__ void dc_conv(const DeltaParams& p, const float* hist, int c, int col, int m, int t, int pos, int C, int rows, float (&y)[kDcTok]) {
  const float* cw = p.conv_w + static_cast<size_t>(c) * p.taps;
  float acc[kDcTok];
#pragma unroll
  for (int r = 0; r < kDcTok; ++r) acc[r] = 0.f;
  if constexpr (TAPS > 0) {
    float x[TAPS + kDcTok - 1], w[TAPS];
#pragma unroll
    for (int i = 0; i < TAPS; ++i) w[i] = cw[i];
#pragma unroll
    for (int i = 0; i < TAPS + kDcTok - 1; ++i) {                   // input row m - (TAPS - 1) + i
      const int back = TAPS - 1 - i;
      x[i] = 0.f;
      if (-back < rows) {
        if (back <= t) x[i] = p.x[static_cast<size_t>(m - back) * p.ldx + col];
        else if (back <= pos) x[i] = hist[static_cast<size_t>((pos - back) % TAPS) * C + c];
      }
    }
#pragma unroll
    for (int r = 0; r < kDcTok; ++r)
#pragma unroll
      for (int i = 0; i < TAPS; ++i) acc[r] = fmaf(x[r + i], w[i], acc[r]);
  } else {
    for (int back = p.taps - 1; back > -kDcTok; --back) {           // input row m - back feeds rows r >= -back
      if (-back >= rows) break;
      float x = 0.f;
      if (back <= t) x = p.x[static_cast<size_t>(m - back) * p.ldx + col];
      else if (back <= pos) x = hist[static_cast<size_t>((pos - back) % p.taps) * C + c];
#pragma unroll
      for (int r = 0; r < kDcTok; ++r) {
        const int i = p.taps - 1 - (r + back);                      // tap of this input for row r
        if (i >= 0 && i < p.taps) acc[r] = fmaf(x, cw[i], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kDcTok; ++r) y[r] = r < rows ? silu_f32(acc[r]) : 0.f;
}

// grid (slots, HK), 256 threads
template <int TAPS>
__global__ void __launch_bounds__(256) delta_chunk_prep_kernel(const __grid_constant__ DeltaParams p) {
  pdl_wait();
  extern __shared__ __align__(16) float dc_sm[];    // k [16][DP + 4] | q [16][DP + 4]
  __shared__ float kk_s[kDcTok][kDcTok + 1], kq_s[kDcTok][kDcTok + 1], a_s[8][kDcTok][kDcTok + 1], g_s[8][kDcTok], b_s[8][kDcTok];
  int j = 0, c = 0;
  bool found = false;
  for (; j < p.nseq; ++j) {
    const int r0 = p.cu_rows[j], n = p.cu_rows[j + 1] - r0;
    c = static_cast<int>(blockIdx.x) - dc_slot(r0, j);
    if (c >= 0 && c * kDcTok < n) { found = true; break; }
  }
  if (!found) return;
  const int slot = dc_state_slot(p, j);
  if (slot < 0) return;
  const int DP = p.DP, ld = DP + 4, hk = blockIdx.y, group = p.H / p.HK, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = c * kDcTok, m = p.cu_rows[j] + t, rows = min(kDcTok, p.cu_rows[j + 1] - m), pos = p.pos[m];
  const int C = 2 * p.HK * p.D + p.H * p.V;
  const float* hist = p.hist + static_cast<size_t>(slot) * p.taps * C;
  const DcLayout lay = dc_layout(p.H, p.HK, DP, p.VP);
  uint8_t* base = reinterpret_cast<uint8_t*>(p.chunk) + blockIdx.x * lay.bytes;
  // ---- keys and queries
  for (int i = threadIdx.x; i < 2 * DP; i += 256) {
    const int isq = i >= DP ? 1 : 0, d = i - isq * DP;
    float y[kDcTok];
#pragma unroll
    for (int r = 0; r < kDcTok; ++r) y[r] = 0.f;
    if (d < p.D) dc_conv<TAPS>(p, hist, (isq ? hk : p.HK + hk) * p.D + d, (isq ? p.q_off : p.k_off) + hk * p.D + d, m, t, pos, C, rows, y);
#pragma unroll
    for (int r = 0; r < kDcTok; ++r) dc_sm[(isq * kDcTok + r) * ld + d] = y[r];
  }
  // ---- values, sixteen rows of a channel a thread
  const int slices = (p.VP + kDcCols - 1) / kDcCols, wide = slices * kDcCols;
  for (int i = threadIdx.x; i < group * wide; i += 256) {
    const int h = hk * group + i / wide, d = i % wide;
    float y[kDcTok];
#pragma unroll
    for (int r = 0; r < kDcTok; ++r) y[r] = 0.f;
    if (d < p.V) dc_conv<TAPS>(p, hist, 2 * p.HK * p.D + h * p.V + d, p.v_off + h * p.V + d, m, t, pos, C, rows, y);
    float* o = reinterpret_cast<float*>(base + lay.v + (static_cast<size_t>(h) * slices + d / kDcCols) * kDcV) + d % kDcCols;
#pragma unroll
    for (int r = 0; r < kDcTok; ++r) o[r * kDcVRow] = y[r];
  }
  __syncthreads();
  // ---- unit norms; the parts of keys and queries
  uint8_t* rec = base + static_cast<size_t>(hk) * dc_kq(DP);
  for (int v = warp; v < 2 * kDcTok; v += 8) {
    float* x = dc_sm + v * ld;
    float sq = 0.f;
    for (int d = lane * 4; d < DP; d += 128) {
      const float4 f = *reinterpret_cast<const float4*>(x + d);
      sq += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
    }
    const bool isq = v >= kDcTok;
    const float s = 1.f / sqrtf(warp_sum_f(sq) + p.unit_eps) * (isq ? p.q_scale : 1.f);
    uint8_t* d0 = rec + (isq ? 3 : 0) * kDcTok * DP * 2;
    for (int d = lane * 4; d < DP; d += 128) {
      float4 f = *reinterpret_cast<const float4*>(x + d);
      f = make_float4(f.x * s, f.y * s, f.z * s, f.w * s);
      *reinterpret_cast<float4*>(x + d) = f;
      uint32_t a[3], b[3];
      dc_split(f.x, f.y, a[0], a[1], a[2]);
      dc_split(f.z, f.w, b[0], b[1], b[2]);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(d0 + e * kDcTok * DP * 2 + dc_at(v & (kDcTok - 1), d)) = make_uint2(a[e], b[e]);
    }
  }
  // ---- decays and rates of the group's value heads
  const int heads = min(group, 8);
  for (int h0 = 0; h0 < group; h0 += heads) {
    const int nh = min(heads, group - h0);
    for (int i = threadIdx.x; i < nh * kDcTok; i += 256) {
      const int h = hk * group + h0 + i / kDcTok, r = i % kDcTok;
      float beta = 0.f, g = 1.f;
      if (r < rows) {
        const float* x = p.x + static_cast<size_t>(m + r) * p.ldx;
        beta = sigmoid_f32(x[p.b_off + h]);
        g = expf(-expf(p.A_log[h]) * softplus_f32(x[p.a_off + h] + p.dt_bias[h]));
      }
      b_s[i / kDcTok][r] = beta;
      g_s[i / kDcTok][r] = g;
    }
    __syncthreads();
    if (h0 == 0) {                                  // dot products of the chunk's tokens: a thread per pair
      const int i = threadIdx.x >> 4, jj = threadIdx.x & 15;
      if (jj <= i) {
        const float *kj = dc_sm + jj * ld, *ki = dc_sm + i * ld, *qi = dc_sm + (kDcTok + i) * ld;
        float kk[16] = {}, kq[16] = {};             // (sixteen short sums: one of 128 terms rounds more than the four-token scan's tree did)
        for (int d = 0; d < DP; d += 16)
#pragma unroll
          for (int u = 0; u < 16; u += 4) {
            const float4 a = *reinterpret_cast<const float4*>(kj + d + u), b = *reinterpret_cast<const float4*>(ki + d + u), q = *reinterpret_cast<const float4*>(qi + d + u);
            kk[u] = fmaf(a.x, b.x, kk[u]); kk[u + 1] = fmaf(a.y, b.y, kk[u + 1]); kk[u + 2] = fmaf(a.z, b.z, kk[u + 2]); kk[u + 3] = fmaf(a.w, b.w, kk[u + 3]);
            kq[u] = fmaf(a.x, q.x, kq[u]); kq[u + 1] = fmaf(a.y, q.y, kq[u + 1]); kq[u + 2] = fmaf(a.z, q.z, kq[u + 2]); kq[u + 3] = fmaf(a.w, q.w, kq[u + 3]);
          }
#pragma unroll
        for (int w = 8; w > 0; w >>= 1)
#pragma unroll
          for (int u = 0; u < w; ++u) {
            kk[u] += kk[u + w];
            kq[u] += kq[u + w];
          }
        kk_s[i][jj] = kk[0];
        kq_s[i][jj] = kq[0];
      }
      __syncthreads();
    }
    for (int e = warp; e < nh; e += 8) {            // a warp per value head, lanes 0 .. 15
      const int h = hk * group + h0 + e;
      uint8_t* sr = base + lay.small + static_cast<size_t>(h) * kDcSmall;
      if (lane < kDcTok) {
        const int i = lane;
        const float beta = b_s[e][i];
        DcProduct d, end;
        for (int jj = kDcTok - 1; jj >= 0; --jj) {  // D_ij, row i
          const bool in = jj <= i;
          if (in && jj < i) a_s[e][i][jj] = beta * d.value() * kk_s[i][jj];
          dc_store_part3(sr + kDcMat, i, jj, in ? d.value() * kq_s[i][jj] : 0.f);
          if (in) d.times(g_s[e][jj]);
          if (jj > i) end.times(g_s[e][jj]);
        }
        float* co = reinterpret_cast<float*>(sr + 2 * kDcMat);
        co[i] = beta;
        co[kDcTok + i] = beta * d.value();
        co[2 * kDcTok + i] = d.value();                     // (d went through all of g_1 .. g_i)
        co[3 * kDcTok + i] = end.value();
      }
      __syncwarp();
      if (lane < kDcTok) {                          // column `lane` of T, without its diagonal of ones
        float x[kDcTok];
#pragma unroll
        for (int i = 0; i < kDcTok; ++i) {
          float s = i == lane ? 1.f : 0.f;
#pragma unroll
          for (int jj = 0; jj < i; ++jj) s = fmaf(-a_s[e][i][jj], x[jj], s);
          x[i] = i < lane ? 0.f : s;
          dc_store_part3(sr, i, lane, i == lane ? 0.f : x[i]);
        }
      }
      __syncwarp();
    }
    __syncthreads();                                // (the gates and rows are reused)
  }
}

// grid (nseq, H, ceil(VP / 32)).  NJ: 64-wide blocks of the key size.
template <int NJ>
__global__ void __launch_bounds__(kDcThreads) delta_chunk_scan_kernel(const __grid_constant__ DeltaParams p) {
  constexpr int DP = NJ * 64, kKS = DP / 32;        // 16-wide key steps of a warp (half of the keys)
  constexpr uint32_t kKq = dc_kq(DP), kPart = kDcTok * DP * 2, kStage = (kKq + kDcV + kDcSmall + 127) / 128 * 128;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[2 * kDcStages];
  __shared__ float4 half_s[2][2][2][3][32];         // [parity of the chunk][pair][half][tiles][lane]: the other warp may still read the last chunk's
  __shared__ volatile uint32_t abort_s[2];
  pdl_wait();
  const int j = blockIdx.x, h = blockIdx.y;
  const int r0 = p.cu_rows[j], n = p.cu_rows[j + 1] - r0;
  if (n <= 0) return;
  const int slot = dc_state_slot(p, j);
  if (slot < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (n + kDcTok - 1) / kDcTok, slices = (p.VP + kDcCols - 1) / kDcCols, hk = h / (p.H / p.HK);
  const uint32_t st0 = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint8_t* const gen = smem_raw + (st0 - smem_u32(smem_raw));
  const uint32_t full = smem_u32(bars), empty = full + 8 * kDcStages;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kDcStages; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 4);
    }
    abort_s[0] = abort_s[1] = 0u;
    mbar_init_fence();
  }
  __syncthreads();
  if (warp == 4) {                                  // ---- copies
    if (lane == 0) {
      const DcLayout lay = dc_layout(p.H, p.HK, DP, p.VP);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(p.chunk) + static_cast<size_t>(dc_slot(r0, j)) * lay.bytes;
      const size_t at_kq = static_cast<size_t>(hk) * kKq, at_v = lay.v + (static_cast<size_t>(h) * slices + blockIdx.z) * kDcV, at_s = lay.small + static_cast<size_t>(h) * kDcSmall;
      int c = 0;
      for (; c < chunks; ++c, src += lay.bytes) {
        const int s = c % kDcStages;
        if (c >= kDcStages && !mbar_wait(empty + 8 * s, ((c / kDcStages) & 1) ^ 1, p.err, kErrWaitEmpty)) break;
        const uint32_t dst = st0 + s * kStage, b = full + 8 * s;
        mbar_arrive_expect_tx(b, kKq + kDcV + kDcSmall);
        bulk_g2s(dst, src + at_kq, kKq, b);
        bulk_g2s(dst + kKq, src + at_v, kDcV, b);
        bulk_g2s(dst + kKq + kDcV, src + at_s, kDcSmall, b);
      }
      for (int i = max(0, c - kDcStages); i < c; ++i)               // the CTA does not leave before its copies have landed
        mbar_wait(full + 8 * (i % kDcStages), (i / kDcStages) & 1, p.err, kErrWaitDrain);
    }
    return;
  }
  const int wv = warp & 1, hn = warp >> 1, q2 = (lane & 3) * 2, l4 = lane >> 2;
  const int v0 = blockIdx.z * kDcCols + wv * 16;
  // this warp's value columns and keys: S[8 keys][column l4 | + 8, keys q2 + {0, 1}]
  float S[2 * kKS][4];
  float* st = p.state + ((static_cast<size_t>(slot) * p.H + h) * p.VP + v0) * DP + hn * (DP / 2);
#pragma unroll
  for (int t = 0; t < 2 * kKS; ++t)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int v = l4 + half * 8;
      const float2 f = v0 + v < p.VP ? *reinterpret_cast<const float2*>(st + static_cast<size_t>(v) * DP + t * 8 + q2) : make_float2(0.f, 0.f);
      S[t][half * 2] = f.x;
      S[t][half * 2 + 1] = f.y;
    }
  const int tr = (lane & 7) + ((lane >> 4) << 3), tc = (lane >> 3) & 1;       // row and column piece of this lane in a 16 x 16 block, rows as columns of the operand
  bool ok = true;
  for (int c = 0; c < chunks; ++c) {
    const int s = c % kDcStages;
    // (both warps of a pair leave together: one that gives up is counted at their next meeting)
    ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, (c / kDcStages) & 1, p.err, kErrWaitFull));
    if (!ok) {
      abort_s[wv] = 1u;
      __threadfence_block();
      named_bar_arrive(1 + wv, 64);
      break;
    }
    const uint32_t kt = st0 + s * kStage, qt = kt + 3 * kPart, mats = kt + kKq + kDcV;
    const float* vt = reinterpret_cast<const float*>(gen + s * kStage + kKq) + wv * 16;
    const float* co = reinterpret_cast<const float*>(gen + s * kStage + kKq + kDcV + 2 * kDcMat);
    // ---- S_0^T k and S_0^T q over this warp's keys
    float pk[2][2][4] = {}, pq[2][2][4] = {};
#pragma unroll
    for (int ks = 0; ks < kKS; ++ks) {
      uint32_t a[3][4], bk[3][4], bq[3][4];
      dc_operand(S[2 * ks], S[2 * ks + 1], a);
      const int ch = (hn * kKS + ks) * 2 + tc;                      // 8-channel piece
      const uint32_t at = static_cast<uint32_t>((ch >> 3) * kDcTok * 128 + tr * 128 + (((ch ^ tr) & 7) << 4));
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        ldsm4(bk[e], kt + e * kPart + at);
        ldsm4(bq[e], qt + e * kPart + at);
      }
      dc_mma6_apart<2>(pk, pq, a, bk, bq);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        pk[0][i][e] += pk[1][i][e];
        pq[0][i][e] += pq[1][i][e];
      }
    // ---- the halves meet: all of the keys' products, one token tile of the queries' each
    half_s[c & 1][wv][hn][0][lane] = make_float4(pk[0][0][0], pk[0][0][1], pk[0][0][2], pk[0][0][3]);
    half_s[c & 1][wv][hn][1][lane] = make_float4(pk[0][1][0], pk[0][1][1], pk[0][1][2], pk[0][1][3]);
    {
      const float (&o)[4] = hn == 0 ? pq[0][1] : pq[0][0];
      half_s[c & 1][wv][hn][2][lane] = make_float4(o[0], o[1], o[2], o[3]);
    }
    named_bar_sync(1 + wv, 64);
    if (abort_s[wv] != 0u) { ok = false; break; }
    const float4 x0 = half_s[c & 1][wv][hn ^ 1][0][lane], x1 = half_s[c & 1][wv][hn ^ 1][1][lane], x2 = half_s[c & 1][wv][hn ^ 1][2][lane];
    const float other[2][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}};
    float X[2][4], mine[4] = {x2.x, x2.y, x2.z, x2.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) mine[e] += hn == 0 ? pq[0][0][e] : pq[0][1][e];
    // ---- beta (v - G S_0^T k)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int tok = i * 8 + q2;
      const float2 be = *reinterpret_cast<const float2*>(co + tok), bg = *reinterpret_cast<const float2*>(co + kDcTok + tok);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v = vt[(tok + (e & 1)) * kDcVRow + l4 + (e >> 1) * 8];
        const float pe = pk[0][i][e] + other[i][e];
        X[i][e] = fmaf(e & 1 ? be.y : be.x, v, -(e & 1 ? bg.y : bg.x) * pe);
      }
    }
    // ---- u = T X (the diagonal of ones: X itself, exact)
    float U[2][4] = {};
    {
      uint32_t a[3][4], b[3][4];
      dc_operand(X[0], X[1], a);
#pragma unroll
      for (int e = 0; e < 3; ++e) ldsm4(b[e], mats + e * 16 * kDcPairRow + tr * kDcPairRow + tc * 16);
      dc_mma6<2>(U, a, b);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) U[i][e] += X[i][e];
    }
    // ---- read-out of this warp's eight tokens
    {
      uint32_t a[3][4], b[3][2];
      dc_operand(U[0], U[1], a);
      const uint32_t row = mats + kDcMat + (hn * 8 + (lane & 7)) * kDcPairRow + ((lane >> 3) & 1) * 16;
#pragma unroll
      for (int e = 0; e < 3; ++e)
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b[e][0]), "=r"(b[e][1]) : "r"(row + e * 16 * kDcPairRow));
      float o[1][4] = {};
      dc_mma6<1>(o, a, b);
      const int tok = hn * 8 + q2;
      const float2 g = *reinterpret_cast<const float2*>(co + 2 * kDcTok + tok);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int v = v0 + l4 + (e >> 1) * 8, i = c * kDcTok + tok + (e & 1);
        if (i < n && v < p.VP) p.o[(static_cast<size_t>(r0 + i) * p.H + h) * p.VP + v] = fmaf(e & 1 ? g.y : g.x, mine[e], o[0][e]);
      }
    }
    // ---- state at the chunk's end
    {
      uint32_t a[3][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 d = *reinterpret_cast<const float2*>(co + 3 * kDcTok + i * 8 + q2);
#pragma unroll
        for (int e = 0; e < 4; ++e) U[i][e] *= e & 1 ? d.y : d.x;
      }
      dc_operand(U[0], U[1], a);
      const float G = co[3 * kDcTok - 1];
#pragma unroll
      for (int ks = 0; ks < kKS; ks += 2) {        // (an even number of steps)
        uint32_t b[2][3][4];
        const int r = lane & 15;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int ch = (hn * kKS + ks + u) * 2 + (lane >> 4);
          const uint32_t at = static_cast<uint32_t>((ch >> 3) * kDcTok * 128 + r * 128 + (((ch ^ r) & 7) << 4));
#pragma unroll
          for (int e = 0; e < 3; ++e) ldsm4_t(b[u][e], kt + e * kPart + at);
        }
        float d[2][2][4] = {};
        dc_mma6<2, 2>(d[0], a, b[0], d[1], a, b[1]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[2 * (ks + u) + i][e] = fmaf(G, S[2 * (ks + u) + i][e], d[u][i][e]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * s);      // this warp is done with the stage
  }
  if (!ok) return;
#pragma unroll
  for (int t = 0; t < 2 * kKS; ++t)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int v = l4 + half * 8;
      if (v0 + v < p.VP) *reinterpret_cast<float2*>(st + static_cast<size_t>(v) * DP + t * 8 + q2) = make_float2(S[t][half * 2], S[t][half * 2 + 1]);
    }
}

template <int NJ>
static int dc_go(const DeltaParams& p, cudaStream_t stream) {
  constexpr int DP = NJ * 64, smem = kDcStages * ((dc_kq(DP) + kDcV + kDcSmall + 127) / 128 * 128) + 128;
  static bool ready[64];
  int e = dc_allow(delta_chunk_scan_kernel<NJ>, ready, smem);
  if (e != 0) return e;
  const dim3 grid(p.M / kDcTok + p.nseq, p.HK);
  const int prep = 2 * kDcTok * (DP + 4) * 4;
  e = static_cast<int>(p.taps == 4 ? launch(delta_chunk_prep_kernel<4>, grid, dim3(256), prep, stream, 0, p) : launch(delta_chunk_prep_kernel<0>, grid, dim3(256), prep, stream, 0, p));
  if (e != 0) return e;
  return static_cast<int>(launch(delta_chunk_scan_kernel<NJ>, dim3(p.nseq, p.H, (p.VP + kDcCols - 1) / kDcCols), dim3(kDcThreads), smem, stream, 0, p));
}

}  // namespace saber

// Scratch of the chunk form in floats (0: it does not take these sizes).
extern "C" size_t saber_delta_chunk_floats(const saber::DeltaParams* p) {
  if (p->DP > 256 || (p->DP & 63) || p->HK <= 0 || p->H % p->HK) return 0;
  return (static_cast<size_t>(p->M) / saber::kDcTok + p->nseq) * saber::dc_layout(p->H, p->HK, p->DP, p->VP).bytes / 4;
}
int saber_delta_chunk_launch(const saber::DeltaParams* p, cudaStream_t stream) {
  switch (p->DP) {
    case 64: return saber::dc_go<1>(*p, stream);
    case 128: return saber::dc_go<2>(*p, stream);
    case 192: return saber::dc_go<3>(*p, stream);
    case 256: return saber::dc_go<4>(*p, stream);
    default: return static_cast<int>(cudaErrorInvalidValue);
  }
}
