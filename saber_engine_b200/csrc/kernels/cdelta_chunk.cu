// Delta rule with a decay and a removal rate per key channel over prompt portions on the tensor cores: sixteen tokens at a time, the state in
// registers.
//
// With c_i = w_1 .. w_i (channel by channel from the chunk's start), b_i = -rate_i u_i and p_i = u_i^T S_{i-1},
//     U_i = u_i c_{i-1},  R_i = r_i c_i,  K_j = k_j / c_j,  B_j = b_j / c_j
//     p = T (U S_0 + (U . K below the diagonal) v),   T = (1 - (U . B below the diagonal))^-1
//     o = R S_0 + (R . K) v + (R . B) p               (on and below the diagonal)
//     S = c_16 (S_0 + K^T v + B^T p)
// A decay is exp(-exp(-1/2) sigmoid(.)), never below 0.545: sixteen of them stay above 6e-5, so that the quotients cost range, of which fp32 and
// bf16 have plenty, and no digits (every term is a product, and its relative error a few units in the last place).
//
//   prep   a CTA per (chunk, four heads): decays (W2 tanh(l) as in cdelta.cu), the four matrices in three bf16 parts (chunk16.cuh), their dot
//          products by `mma.sync`, T by forward substitution
//   scan   a CTA per (sequence, head, 32 value columns), as in delta_chunk.cu: two pairs of warps, sixteen columns a pair, half of the keys a warp
// Bound by the chain of dependent products a chunk (scan) and by the parts' conversions and W2 products (preparation).  2048 tokens, 32 heads of 128 x 128:
// scan 213 us (blocks of four tokens: 457), preparation 217 (151).  Error against 64 bits over 37 to 2048 tokens: 0.16 to 1.4e-6 of the output and
// 0.2 to 1.5e-6 of the state, the four-token scan's 0.2 to 1.5e-6 and 0.25 to 1.6e-6.
#include "cdelta.h"
#include "chunk16.cuh"
#include "launch.cuh"
#include "scan_records.cuh"

namespace saber {

constexpr float kCcRate = 0.60653065971263342f;     // exp(-1/2)
constexpr int kCcHeads = 4, kCcRank = 256;
__host__ __device__ constexpr int cc_part(int DP) { return kDcTok * DP * 2; }
__host__ __device__ constexpr int cc_mats(int DP) { return 12 * cc_part(DP); }                         // U | R | K | B, three parts each
__host__ __device__ constexpr int cc_small(int DP) { return 4 * kDcMat + DP * 4; }                    // U . K | T | R . K | R . B | c_16
__host__ __device__ inline size_t cc_record(int DP, int VP) { return static_cast<size_t>(cc_mats(DP) + cc_small(DP)) + static_cast<size_t>((VP + kDcCols - 1) / kDcCols) * kDcV; }
__host__ __device__ constexpr int cc_rank_pad(int rank) { return (rank + 15) & ~15; }

__device__ __forceinline__ int cc_state_slot(const CdeltaParams& p, int j) {
  const int s = p.slots[j];
  if (s >= p.n_slots) {
    if (p.err) atomicCAS(p.err, 0u, static_cast<uint32_t>(kErrBadIndex));
    return -1;
  }
  return s;
}

// grid (slots, ceil(H / 4)), DP threads (a channel each).  Shared memory: matrices | tanh(l) in three parts [3][16][RK + 8] | products [16][DP + 4].
template <int DP>
__global__ void __launch_bounds__(DP, DP == 128 ? 3 : 5) cdelta_chunk_prep_kernel(const __grid_constant__ CdeltaParams p) {
  pdl_wait();
  constexpr int kWarps = DP / 32, ZS = DP + 4, kPart = cc_part(DP), NI = DP / 8 / kWarps;      // NI: 8-channel tiles of a warp
  extern __shared__ __align__(128) uint8_t cc_sm[];
  __shared__ float red[kWarps][kDcTok], ub_s[kCcHeads][kDcTok][kDcTok + 1];
  int j = 0, c = 0;
  bool found = false;
  for (; j < p.nseq; ++j) {
    const int r0 = p.cu_rows[j], n = p.cu_rows[j + 1] - r0;
    c = static_cast<int>(blockIdx.x) - dc_slot(r0, j);
    if (c >= 0 && c * kDcTok < n) { found = true; break; }
  }
  if (!found || cc_state_slot(p, j) < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = threadIdx.x, RK = cc_rank_pad(p.rank);
  const int m = p.cu_rows[j] + c * kDcTok, rows = min(kDcTok, p.cu_rows[j + 1] - m);
  const float* x = p.x + static_cast<size_t>(m) * p.ldx;
  const uint32_t ms = smem_u32(cc_sm), ts = ms + cc_mats(DP), t_row = static_cast<uint32_t>(RK + 8) * 2u, t_part = 16u * t_row;
  float* zs = reinterpret_cast<float*>(cc_sm + cc_mats(DP) + 3 * t_part);
  const size_t rec_bytes = cc_record(DP, p.VP);
  for (int i = threadIdx.x; i < kDcTok * RK; i += DP) {
    const int r = i / RK, q = i - r * RK;
    float t = r < rows && q < p.rank ? tanhf(x[static_cast<size_t>(r) * p.ldx + p.l_off + q]) : 0.f;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      const __nv_bfloat16 v = __float2bfloat16(t);
      asm volatile("st.shared.b16 [%0], %1;" ::"r"(ts + part * t_part + r * t_row + q * 2), "h"(__bfloat16_as_ushort(v)) : "memory");
      t -= __bfloat162float(v);
    }
  }
  const uint32_t a_row = ts + static_cast<uint32_t>(lane & 15) * t_row + ((lane >> 4) << 4);
  const __nv_bfloat16* w2 = static_cast<const __nv_bfloat16*>(p.w2);
  const int q2 = (lane & 3) * 2, l4 = lane >> 2, tr = (lane & 7) + ((lane >> 4) << 3), tc = (lane >> 3) & 1;
  const bool in = d < p.D;
  const int h1 = min(p.H, (static_cast<int>(blockIdx.y) + 1) * kCcHeads);
  {                                                 // values as they are
    const int slices = (p.VP + kDcCols - 1) / kDcCols;
    if (d < slices * kDcCols)
      for (int h = blockIdx.y * kCcHeads; h < h1; ++h) {
        uint8_t* rec = reinterpret_cast<uint8_t*>(p.chunk) + (static_cast<size_t>(blockIdx.x) * p.H + h) * rec_bytes;
        float* o = reinterpret_cast<float*>(rec + cc_mats(DP) + cc_small(DP) + static_cast<size_t>(d / kDcCols) * kDcV) + d % kDcCols;
        float v[kDcTok];
#pragma unroll
        for (int i = 0; i < kDcTok; ++i) v[i] = x[static_cast<size_t>(min(i, rows - 1)) * p.ldx + p.v_off + h * p.D + (in ? d : 0)];
#pragma unroll
        for (int i = 0; i < kDcTok; ++i) o[i * kDcVRow] = in && i < rows ? v[i] : 0.f;
      }
  }
  // this channel's projections, requested a head ahead
  float k[kDcTok], a[kDcTok], r[kDcTok];
  auto request = [&](int h) {
#pragma unroll
    for (int i = 0; i < kDcTok; ++i) {
      const float* xi = x + static_cast<size_t>(min(i, rows - 1)) * p.ldx + h * p.D + (in ? d : 0);
      k[i] = xi[p.k_off];
      a[i] = xi[p.a_off];
      r[i] = xi[p.r_off];
    }
  };
  request(blockIdx.y * kCcHeads);
  for (int h = blockIdx.y * kCcHeads; h < h1; ++h) {
    uint8_t* rec = reinterpret_cast<uint8_t*>(p.chunk) + (static_cast<size_t>(blockIdx.x) * p.H + h) * rec_bytes;
    const int col = h * p.D + (in ? d : 0);
    const float w0 = p.w0[col];
    __syncthreads();                                // (tanh is there; the products and matrices of the head before are read)
    {                                               // W2 tanh(l), NI tiles of eight channels a warp
      float acc[NI][4] = {};
      const __nv_bfloat16* wr[NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int ch = (warp * NI + i) * 8 + l4;
        wr[i] = w2 + static_cast<size_t>(h * p.D + (ch < p.D ? ch : 0)) * RK + q2;
      }
      uint32_t nb[2][NI][2];                         // the next two steps' pieces of W2
      auto fetch = [&](uint32_t (&to)[NI][2], int k0) {
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          to[i][0] = *reinterpret_cast<const uint32_t*>(wr[i] + k0);
          to[i][1] = *reinterpret_cast<const uint32_t*>(wr[i] + k0 + 8);
        }
      };
      auto step = [&](const uint32_t (&b)[NI][2], int k0) {
        uint32_t t[3][4];
#pragma unroll
        for (int part = 0; part < 3; ++part) ldsm4(t[part], a_row + part * t_part + k0 * 2);
#pragma unroll
        for (int part = 2; part >= 0; --part)        // (channels past the head: numbers that nothing reads)
#pragma unroll
          for (int i = 0; i < NI; ++i) mma16816(acc[i], t[part], b[i][0], b[i][1]);
      };
      fetch(nb[0], 0);
      if (RK > 16) fetch(nb[1], 16);
      for (int k0 = 0; k0 < RK; k0 += 32) {
        uint32_t b[NI][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (k0 + 16 * u >= RK) break;
#pragma unroll
          for (int i = 0; i < NI; ++i) { b[i][0] = nb[u][i][0]; b[i][1] = nb[u][i][1]; }
          if (k0 + 16 * u + 32 < RK) fetch(nb[u], k0 + 16 * u + 32);
          step(b, k0 + 16 * u);
        }
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        float* z = zs + l4 * ZS + (warp * NI + i) * 8 + q2;
        *reinterpret_cast<float2*>(z) = make_float2(acc[i][0], acc[i][1]);
        *reinterpret_cast<float2*>(z + 8 * ZS) = make_float2(acc[i][2], acc[i][3]);
      }
    }
    {                                               // |k|^2 of the sixteen tokens: lane n of a warp gets token n's sum
      float v[kDcTok];
#pragma unroll
      for (int i = 0; i < kDcTok; ++i) {
        if (!in || i >= rows) k[i] = 0.f;
        v[i] = k[i] * k[i];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int e = 0; e < o; ++e) {
          const float keep = up ? v[o + e] : v[e], give = up ? v[e] : v[o + e];
          v[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
      if (lane < kDcTok) red[warp][lane] = v[0];
    }
    // the matrices of the head before have left shared memory
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    {
      float unit = 0.f;                  // lane i & 15: of token i
#pragma unroll
      for (int w = 0; w < kWarps; ++w) unit += red[w][lane & (kDcTok - 1)];
      unit = 1.f / sqrtf(unit + p.unit_eps);
      DcProduct cum;
#pragma unroll
      for (int i = 0; i < kDcTok; ++i) {
        const bool live = in && i < rows;
        const float u = k[i] * __shfl_sync(0xffffffffu, unit, i), b = -sigmoid_f32(a[i]) * u;
        const float w = live ? expf(-kCcRate * sigmoid_f32(zs[i * ZS + d] + w0)) : 1.f;
        float f[4];
        f[0] = u * cum.value();
        cum.times(w);
        f[1] = live ? r[i] * cum.value() : 0.f;
        const float inv = __frcp_rn(cum.value());
        f[2] = k[i] * inv;
        f[3] = b * inv;
#pragma unroll
        for (int mat = 0; mat < 4; ++mat) {
          float v = f[mat];
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const __nv_bfloat16 t = __float2bfloat16(v);
            asm volatile("st.shared.b16 [%0], %1;" ::"r"(ms + (mat * 3 + e) * kPart + dc_at(i, d)), "h"(__bfloat16_as_ushort(t)) : "memory");
            v -= __bfloat162float(t);
          }
        }
      }
      reinterpret_cast<float*>(rec + cc_mats(DP) + 4 * kDcMat)[d] = cum.value();
    }
    if (h + 1 < h1) request(h + 1);
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(rec), "r"(ms), "r"(static_cast<uint32_t>(cc_mats(DP))) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    // ---- dot products: U . B first (T waits for it)
    for (int g = warp; g < 4; g += kWarps) {         // U . B, U . K, R . K, R . B
      const uint32_t ma = ms + (g >> 1) * 3 * kPart, mb = ms + (g == 1 || g == 2 ? 2 : 3) * 3 * kPart;
      float acc[3][2][4] = {};
#pragma unroll
      for (int ks = 0; ks < DP / 16; ++ks) {
        uint32_t fa[3][4], fb[3][4];
        const int ar = lane & 15, ac = ks * 2 + (lane >> 4), bc = ks * 2 + tc;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          ldsm4(fa[e], ma + e * kPart + (ac >> 3) * kDcTok * 128 + ar * 128 + (((ac ^ ar) & 7) << 4));
          ldsm4(fb[e], mb + e * kPart + (bc >> 3) * kDcTok * 128 + tr * 128 + (((bc ^ tr) & 7) << 4));
        }
        dc_mma6_apart<2>(acc[0], acc[1 + (ks & 1)], fa, fb);
      }
      uint8_t* to = rec + cc_mats(DP) + (g < 2 ? g ^ 1 : g) * kDcMat;
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int i = l4 + half * 8, jj = n * 8 + q2, reach = g < 2 ? i : i + 1;
          const float y0 = jj < reach ? acc[0][n][half * 2] + (acc[1][n][half * 2] + acc[2][n][half * 2]) : 0.f, y1 = jj + 1 < reach ? acc[0][n][half * 2 + 1] + (acc[1][n][half * 2 + 1] + acc[2][n][half * 2 + 1]) : 0.f;
          if (g == 0) {
            ub_s[h & (kCcHeads - 1)][i][jj] = y0;
            ub_s[h & (kCcHeads - 1)][i][jj + 1] = y1;
          } else {
            uint32_t s[3];
            dc_split(y0, y1, s[0], s[1], s[2]);
#pragma unroll
            for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(to + e * 16 * kDcPairRow + i * kDcPairRow + jj * 2) = s[e];
          }
        }
    }
  }
  // ---- T without its diagonal of ones, a head a warp: column `lane` by a lane
  __syncthreads();
  for (int h = blockIdx.y * kCcHeads + warp; h < h1; h += kWarps)
    if (lane < kDcTok) {
      const float (*ub)[kDcTok + 1] = ub_s[h & (kCcHeads - 1)];
      uint8_t* to = reinterpret_cast<uint8_t*>(p.chunk) + (static_cast<size_t>(blockIdx.x) * p.H + h) * rec_bytes + cc_mats(DP) + kDcMat;
      float t[kDcTok];
#pragma unroll
      for (int i = 0; i < kDcTok; ++i) {
        float s = i == lane ? 1.f : 0.f;
#pragma unroll
        for (int jj = 0; jj < i; ++jj) s = fmaf(ub[i][jj], t[jj], s);
        t[i] = i < lane ? 0.f : s;
        dc_store_part3(to, i, lane, i == lane ? 0.f : t[i]);
      }
    }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// grid (nseq, H, ceil(VP / 32)).  NJ: 64-wide blocks of the key size.
template <int NJ>
__global__ void __launch_bounds__(kDcThreads) cdelta_chunk_scan_kernel(const __grid_constant__ CdeltaParams p) {
  constexpr int DP = NJ * 64, kKS = DP / 32;        // 16-wide key steps of a warp (half of the keys)
  constexpr uint32_t kPart = cc_part(DP), kFixed = cc_mats(DP) + cc_small(DP), kStage = (kFixed + kDcV + 127) / 128 * 128;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[2 * kDcStages];
  __shared__ float4 half_s[2][2][2][3][32];         // [parity of the chunk][pair][half][tiles][lane]: the other warp may still read the last chunk's
  __shared__ volatile uint32_t abort_s[2];
  pdl_wait();
  const int j = blockIdx.x, h = blockIdx.y;
  const int r0 = p.cu_rows[j], n = p.cu_rows[j + 1] - r0;
  if (n <= 0) return;
  const int slot = cc_state_slot(p, j);
  if (slot < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = (n + kDcTok - 1) / kDcTok;
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
      const size_t rec_bytes = cc_record(DP, p.VP);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(p.chunk) + (static_cast<size_t>(dc_slot(r0, j)) * p.H + h) * rec_bytes;
      int c = 0;
      for (; c < chunks; ++c, src += rec_bytes * p.H) {
        const int s = c % kDcStages;
        if (c >= kDcStages && !mbar_wait(empty + 8 * s, ((c / kDcStages) & 1) ^ 1, p.err, kErrWaitEmpty)) break;
        const uint32_t dst = st0 + s * kStage, b = full + 8 * s;
        mbar_arrive_expect_tx(b, kFixed + kDcV);
        bulk_g2s(dst, src, kFixed, b);
        bulk_g2s(dst + kFixed, src + kFixed + static_cast<size_t>(blockIdx.z) * kDcV, kDcV, b);
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
    const uint32_t mt = st0 + s * kStage, sq = mt + cc_mats(DP);
    const float* vt = reinterpret_cast<const float*>(gen + s * kStage + kFixed) + wv * 16;
    const float* c16 = reinterpret_cast<const float*>(gen + s * kStage + cc_mats(DP) + 4 * kDcMat) + hn * (DP / 2);
    // ---- U S_0 and R S_0 over this warp's keys
    float pu[2][2][4] = {}, pr[2][2][4] = {};
#pragma unroll
    for (int ks = 0; ks < kKS; ++ks) {
      uint32_t a[3][4], bu[3][4], br[3][4];
      dc_operand(S[2 * ks], S[2 * ks + 1], a);
      const int ch = (hn * kKS + ks) * 2 + tc;                      // 8-channel piece
      const uint32_t at = static_cast<uint32_t>((ch >> 3) * kDcTok * 128 + tr * 128 + (((ch ^ tr) & 7) << 4));
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        ldsm4(bu[e], mt + e * kPart + at);
        ldsm4(br[e], mt + (3 + e) * kPart + at);
      }
      dc_mma6_apart<2>(pu, pr, a, bu, br);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        pu[0][i][e] += pu[1][i][e];
        pr[0][i][e] += pr[1][i][e];
      }
    // ---- the halves meet: all of U's products, one token tile of R's each
    half_s[c & 1][wv][hn][0][lane] = make_float4(pu[0][0][0], pu[0][0][1], pu[0][0][2], pu[0][0][3]);
    half_s[c & 1][wv][hn][1][lane] = make_float4(pu[0][1][0], pu[0][1][1], pu[0][1][2], pu[0][1][3]);
    {
      const float (&o)[4] = hn == 0 ? pr[0][1] : pr[0][0];
      half_s[c & 1][wv][hn][2][lane] = make_float4(o[0], o[1], o[2], o[3]);
    }
    // ---- what does not wait for them: the values as an operand, (U . K) v, (R . K) v
    uint32_t av[3][4];
    float X[2][4] = {}, o[1][4] = {};
    const uint32_t orow = sq + (hn * 8 + (lane & 7)) * kDcPairRow + ((lane >> 3) & 1) * 16;
    {
      float v[2][4];
      uint32_t b[3][4], b1[3][2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[i][e] = vt[(i * 8 + q2 + (e & 1)) * kDcVRow + l4 + (e >> 1) * 8];
      dc_operand(v[0], v[1], av);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        ldsm4(b[e], sq + e * 16 * kDcPairRow + tr * kDcPairRow + tc * 16);
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b1[e][0]), "=r"(b1[e][1]) : "r"(orow + 2 * kDcMat + e * 16 * kDcPairRow));
      }
      dc_mma6<2, 1>(X, av, b, o, av, b1);
    }
    named_bar_sync(1 + wv, 64);
    if (abort_s[wv] != 0u) { ok = false; break; }
    const float4 x0 = half_s[c & 1][wv][hn ^ 1][0][lane], x1 = half_s[c & 1][wv][hn ^ 1][1][lane], x2 = half_s[c & 1][wv][hn ^ 1][2][lane];
    const float other[2][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}};
    float mine[4] = {x2.x, x2.y, x2.z, x2.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) mine[e] += hn == 0 ? pr[0][0][e] : pr[0][1][e];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) X[i][e] += pu[0][i][e] + other[i][e];
    // ---- p = T X (the diagonal of ones: X itself, exact)
    uint32_t ap[3][4];
    {
      uint32_t a[3][4], b[3][4];
      float P[2][4] = {};
      dc_operand(X[0], X[1], a);
#pragma unroll
      for (int e = 0; e < 3; ++e) ldsm4(b[e], sq + kDcMat + e * 16 * kDcPairRow + tr * kDcPairRow + tc * 16);
      dc_mma6<2>(P, a, b);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) P[i][e] += X[i][e];
      dc_operand(P[0], P[1], ap);
    }
    // ---- state at the chunk's end
#pragma unroll
    for (int ks = 0; ks < kKS; ++ks) {
      uint32_t bk[3][4], bb[3][4];
      const int r = lane & 15, ch = (hn * kKS + ks) * 2 + (lane >> 4);
      const uint32_t at = static_cast<uint32_t>((ch >> 3) * kDcTok * 128 + r * 128 + (((ch ^ r) & 7) << 4));
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        ldsm4_t(bk[e], mt + (6 + e) * kPart + at);
        ldsm4_t(bb[e], mt + (9 + e) * kPart + at);
      }
      float d[2][4] = {}, f[2][4] = {};
      dc_mma6<2, 2>(d, av, bk, f, ap, bb);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 w = *reinterpret_cast<const float2*>(c16 + (2 * ks + i) * 8 + q2);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[2 * ks + i][e] = (e & 1 ? w.y : w.x) * (S[2 * ks + i][e] + (d[i][e] + f[i][e]));
      }
    }
    // ---- read-out of this warp's eight tokens
    {
      uint32_t b[3][2];
#pragma unroll
      for (int e = 0; e < 3; ++e)
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b[e][0]), "=r"(b[e][1]) : "r"(orow + 3 * kDcMat + e * 16 * kDcPairRow));
      float o2[1][4] = {};
      dc_mma6<1>(o2, ap, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int v = v0 + l4 + (e >> 1) * 8, i = c * kDcTok + hn * 8 + q2 + (e & 1);
        if (i < n && v < p.VP) p.o[(static_cast<size_t>(r0 + i) * p.H + h) * p.VP + v] = mine[e] + (o[0][e] + o2[0][e]);
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
static int cc_go(const CdeltaParams& p, cudaStream_t stream) {
  constexpr int DP = NJ * 64, scan = kDcStages * ((cc_mats(DP) + cc_small(DP) + kDcV + 127) / 128 * 128) + 128;
  const int RK = cc_rank_pad(p.rank), prep = cc_mats(DP) + 3 * 16 * (RK + 8) * 2 + kDcTok * (DP + 4) * 4;
  static bool ready[64], ready_prep[64];
  int e = dc_allow(cdelta_chunk_scan_kernel<NJ>, ready, scan);
  if (e == 0) e = dc_allow(cdelta_chunk_prep_kernel<DP>, ready_prep, cc_mats(DP) + 3 * 16 * (kCcRank + 8) * 2 + kDcTok * (DP + 4) * 4);
  if (e == 0) e = static_cast<int>(launch(cdelta_chunk_prep_kernel<DP>, dim3(p.M / kDcTok + p.nseq, (p.H + kCcHeads - 1) / kCcHeads), dim3(DP), prep, stream, 0, p));
  if (e == 0) e = static_cast<int>(launch(cdelta_chunk_scan_kernel<NJ>, dim3(p.nseq, p.H, (p.VP + kDcCols - 1) / kDcCols), dim3(kDcThreads), scan, stream, 0, p));
  return e;
}

}  // namespace saber

// Scratch of the chunk form in floats (0: it does not take these sizes).
extern "C" size_t saber_cdelta_chunk_floats(const saber::CdeltaParams* p) {
  if ((p->DP != 64 && p->DP != 128) || p->w2_f32 || saber::cc_rank_pad(p->rank) > saber::kCcRank) return 0;
  return (static_cast<size_t>(p->M) / saber::kDcTok + p->nseq) * p->H * saber::cc_record(p->DP, p->VP) / 4;
}
int saber_cdelta_chunk_launch(const saber::CdeltaParams* p, cudaStream_t stream) {
  return p->DP == 64 ? saber::cc_go<1>(*p, stream) : p->DP == 128 ? saber::cc_go<2>(*p, stream) : static_cast<int>(cudaErrorInvalidValue);
}
