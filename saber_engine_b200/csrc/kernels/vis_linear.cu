// The vision tower's linears: y = bf16(x W^T + b), then a gelu of it or the residual added to it, each rounded once more.
//
// One tcgen05 kernel over the layouts of the other GEMMs (token rows [k-block of 64][M_pad][128 bytes], weights [256 features][k-block][32 KB],
// both swizzled).  A tower has a few hundred to a few thousand rows, reductions of 18 k-blocks and outputs of 1152 to 4304 features: too small for
// one tile of fixed width per CTA.  So
//   * the width of a tile (64, 128, 192 or 256 features) and the parts its reduction is cut into follow from the shape (vis_linear_shape)
//   * CTAs are resident and walk their tiles; two accumulators in tensor memory let the epilogue of a tile run beside the products of the next
// Bound by the copies of the k-blocks (64 bytes a clock and SM at 256 features).  A block's four linears at 4096 rows: 34 + 18 + 38 + 51 us, 228 in
// the fixed 128 x 256 tiles with row-per-lane stores that this kernel replaces; at 308 rows 10 + 9 + 12 + 18 us, 112 before.
// Parts of a reduction go to a workspace; the last CTA of a tile to arrive adds them in order, so results do not depend on timing.
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "vision.h"

namespace saber {

constexpr int kVlThreads = 320;           // copies, MMA issue, eight epilogue warps
constexpr int kVlStages = 8;
constexpr int kVlSmem = 200 * 1024;       // copies in flight; behind them the epilogue's rows
constexpr int kVlStage = 8 * 32 * 80;

struct VisLinearShape {
  int bn, splits, stages, tiles_n, tiles;
};

__device__ __forceinline__ float vis_gelu_erf(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float vis_gelu_tanh(float x) { return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x))); }

// Finished columns n .. n + 31 of a warp's 32 rows (row `lane` in v): biased, rounded and activated into the warp's part of shared memory, and from
// there by four lanes a row, so that a store fills whole sectors.  4096 x 3456 x 1152, products and copies alone 29 us: 68 with 16 bytes a store and a
// row a lane, 58 staged, 55 with the bias fetched ahead, 34 with one decision a chunk about what is done to its values.
constexpr int kVlRow = kVlStage / 256;    // bytes of a staged row: 32 values and 16 bytes that spread the rows over the banks
__device__ __forceinline__ uint32_t vis_pack2(float a, float b) {
  const __nv_bfloat162 w = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&w);
}
__device__ __forceinline__ uint32_t vis_add2(uint32_t a, uint32_t b) {       // two bf16 sums, rounded once
  const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b));
  return vis_pack2(x.x + y.x, x.y + y.y);
}
struct VlResidual {
  uint4 v[4];
};
__device__ __forceinline__ void vis_linear_residual(const VisLinearParams& p, VlResidual& old, int m0, int n, int lane) {
  if (p.epi != 3 || n + (lane & 3) * 8 + 8 > p.N) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + i * 8 + (lane >> 2);
    if (m < p.M) old.v[i] = *reinterpret_cast<const uint4*>(p.res + static_cast<size_t>(m) * p.ldo + n + (lane & 3) * 8);
  }
}
__device__ __forceinline__ void vis_linear_store(const VisLinearParams& p, const float (&v)[32], const VlResidual& old, const float* bias, uint8_t* stage, int m0, int n, int lane) {
  // (with a decision an element the compiler branches around each of them: 4,500 clocks a chunk)
  float y[32];
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float4 b = *reinterpret_cast<const float4*>(bias + c);
    y[c] = v[c] + b.x;
    y[c + 1] = v[c + 1] + b.y;
    y[c + 2] = v[c + 2] + b.z;
    y[c + 3] = v[c + 3] + b.w;
  }
  if (p.epi == 1) {
#pragma unroll
    for (int c = 0; c < 32; ++c) y[c] = vis_gelu_tanh(__bfloat162float(__float2bfloat16(y[c])));
  } else if (p.epi == 2) {
#pragma unroll
    for (int c = 0; c < 32; ++c) y[c] = vis_gelu_erf(__bfloat162float(__float2bfloat16(y[c])));
  }
#pragma unroll
  for (int c = 0; c < 32; c += 8)
    *reinterpret_cast<uint4*>(stage + lane * kVlRow + c * 2) = make_uint4(vis_pack2(y[c], y[c + 1]), vis_pack2(y[c + 2], y[c + 3]), vis_pack2(y[c + 4], y[c + 5]), vis_pack2(y[c + 6], y[c + 7]));
  __syncwarp();
  const int c = (lane & 3) * 8, left = p.N - n - c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 8 + (lane >> 2), m = m0 + r;
    if (m >= p.M) break;
    uint4 w = *reinterpret_cast<const uint4*>(stage + r * kVlRow + c * 2);
    __nv_bfloat16* o = p.out + static_cast<size_t>(m) * p.ldo + n + c;
    if (left >= 8) {
      if (p.epi == 3) {
        w.x = vis_add2(w.x, old.v[i].x);
        w.y = vis_add2(w.y, old.v[i].y);
        w.z = vis_add2(w.z, old.v[i].z);
        w.w = vis_add2(w.w, old.v[i].w);
      }
      *reinterpret_cast<uint4*>(o) = w;
    } else {
      const __nv_bfloat16* y16 = reinterpret_cast<const __nv_bfloat16*>(&w);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < left) o[j] = p.epi == 3 ? __float2bfloat16(__bfloat162float(y16[j]) + __bfloat162float(p.res[static_cast<size_t>(m) * p.ldo + n + c + j])) : y16[j];
    }
  }
  __syncwarp();                                    // (read before the next columns come)
}

// grid: resident CTAs; item i is part i / tiles of tile i % tiles
__global__ void __launch_bounds__(kVlThreads, 1) vis_linear_kernel(const __grid_constant__ VisLinearParams p, const VisLinearShape sh) {
  pdl_trigger();                                   // (one round of CTAs: the next kernel may get ready beside them; it waits before it reads or writes)
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[2 * kVlStages + 5];
  __shared__ uint32_t tmem_base_s, last_s;
  __shared__ __align__(16) float bias_s[8][128];
  __shared__ volatile uint32_t abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = (p.K + 63) >> 6, per = (KB + sh.splits - 1) / sh.splits, items = sh.tiles * sh.splits;
  const uint32_t abytes = 16384u, wbytes = static_cast<uint32_t>(sh.bn) * 128u;
  const uint32_t a_s = (smem_u32(smem_raw) + 1023u) & ~1023u, w_s = a_s + static_cast<uint32_t>(sh.stages) * abytes;
  const uint32_t full = smem_u32(bars), empty = full + 8 * kVlStages, accfull = empty + 8 * kVlStages, accfree = accfull + 16, bend = accfree + 16;
  const uint32_t cols = sh.bn == 64 ? 128u : sh.bn == 128 ? 256u : 512u;
  if (threadIdx.x == 0) {
    for (int s = 0; s < sh.stages; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accfull + 8 * i, 1);
      mbar_init(accfree + 8 * i, 8);
    }
    mbar_init(bend, 1);
    abort_s = 0u;
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_base_s;

  if (warp == 0) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      const uint64_t keep = l2_policy_evict_normal();
      int s = 0, filled = 0;
      uint32_t ph = 1;
      bool ok = true, waited = false;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        const int tile = item % sh.tiles, kb0 = item / sh.tiles * per, nkb = min(KB, kb0 + per) - kb0;
        const int n0 = tile % sh.tiles_n * sh.bn, m0 = tile / sh.tiles_n * 128;
        const uint32_t arows = static_cast<uint32_t>(min(128, p.M_pad - m0)), wrows = static_cast<uint32_t>(min(sh.bn, p.N_pad - n0));
        auto weights = [&](int kb, int at) {       // rows n0 .. of the 256-row tiles they lie in
          for (uint32_t r = 0; r < wrows;) {
            const uint32_t n = static_cast<uint32_t>(n0) + r, cnt = min(wrows - r, 256u - (n & 255u));
            bulk_g2s_hint(w_s + at * wbytes + r * 128u, p.w + (static_cast<size_t>(n >> 8) * KB + kb) * 32768u + (n & 255u) * 128u, cnt * 128u, full + 8 * at, keep);
            r += cnt;
          }
        };
        int kb = 0;
        if (!waited) {                             // the first stages' weights go out ahead of the wait: no kernel writes them
          const int pre = min(sh.stages, nkb);
          for (int i = 0; i < pre; ++i) {
            mbar_arrive_expect_tx(full + 8 * i, (arows + wrows) * 128u);
            weights(kb0 + i, i);
          }
          pdl_wait();
          waited = true;
          for (int i = 0; i < pre; ++i) bulk_g2s(a_s + i * abytes, p.a + (static_cast<size_t>(kb0 + i) * p.M_pad + m0) * 128, arows * 128u, full + 8 * i);
          kb = filled = pre;
          s = pre == sh.stages ? 0 : pre;
          ph = pre == sh.stages ? 0u : 1u;
        }
        for (; kb < nkb; ++kb) {
          if (filled >= sh.stages && !mbar_wait(empty + 8 * s, ph, p.err, kErrWaitEmpty)) { ok = false; break; }
          mbar_arrive_expect_tx(full + 8 * s, (arows + wrows) * 128u);
          weights(kb0 + kb, s);
          bulk_g2s(a_s + s * abytes, p.a + (static_cast<size_t>(kb0 + kb) * p.M_pad + m0) * 128, arows * 128u, full + 8 * s);
          ++filled;
          if (++s == sh.stages) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok)                                     // do not leave while an own copy is in flight
        for (int i = max(0, filled - sh.stages); i < filled; ++i) mbar_wait(full + 8 * (i % sh.stages), (i / sh.stages) & 1, p.err, kErrWaitDrain);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (elected, and unrolled: issued by a lane number's thread each product costs 90 to 165 clocks)
    if (elect_one()) {
      const uint32_t idesc = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, static_cast<uint32_t>(sh.bn));
      int s = 0, i = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x, ++i) {
        const int kb0 = item / sh.tiles * per, nkb = min(KB, kb0 + per) - kb0, buf = i & 1;
        if (i >= 2 && !mbar_wait(accfree + 8 * buf, ((i >> 1) & 1) ^ 1, p.err, kErrWaitReady)) break;
        tc_fence_after_sync();
        const uint32_t d = tm + static_cast<uint32_t>(buf * sh.bn);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(full + 8 * s, ph, p.err, kErrWaitReady)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t ad = make_desc_k128(a_s + s * abytes), wd = make_desc_k128(w_s + s * wbytes);
#pragma unroll
          for (int j = 0; j < 4; ++j) mma_f16_ss(d, ad + 2 * j, wd + 2 * j, idesc, (kb | j) != 0 ? 1u : 0u);
          mma_commit(empty + 8 * s);
          if (++s == sh.stages) { s = 0; ph ^= 1u; }
        }
        if (ok) mma_commit(accfull + 8 * buf);
      }
      mma_commit(bend);                            // everything issued has retired before the tensor memory goes back
      mbar_wait(bend, 0, p.err, kErrWaitDrain);
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int q4 = warp & 3, half = (warp - 2) >> 2, te = threadIdx.x - 64;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const int chunks = sh.bn / 64;                 // of 32 columns, of this warp's half
    uint8_t* const stage = smem_raw + (a_s - smem_u32(smem_raw)) + sh.stages * (abytes + wbytes) + (warp - 2) * 32 * kVlRow;
    pdl_wait();
    int i = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, ++i) {
      const int tile = item % sh.tiles, split = item / sh.tiles, buf = i & 1;
      const int n0 = tile % sh.tiles_n * sh.bn + half * (sh.bn / 2), m0 = tile / sh.tiles_n * 128;
      const int m = m0 + q4 * 32 + lane;
      const bool live = m < p.M;
      float* const bias = bias_s[warp - 2];          // (requested ahead of the wait: looked up where it is needed it cost a round trip per eight columns)
      for (int c = lane; c < sh.bn / 2; c += 32) bias[c] = p.bias != nullptr && n0 + c < p.N ? p.bias[n0 + c] : 0.f;
      __syncwarp();
      // (decided by the warp as a whole: tensor-memory accesses need all its lanes together)
      if (!__all_sync(0xffffffffu, mbar_wait(accfull + 8 * buf, (i >> 1) & 1, p.err, kErrWaitAcc))) {
        if (sh.splits > 1) {                       // the others meet at a barrier without a time limit: counted there, they leave behind it
          abort_s = 1u;
          __threadfence_block();
          named_bar_arrive(1, 256);
        }
        break;
      }
      tc_fence_after_sync();
      const uint32_t src = tm + static_cast<uint32_t>(buf * sh.bn + half * (sh.bn / 2)) + lane_off;
      for (int c = 0; c < chunks; ++c) {
        uint32_t r[32];
        VlResidual old;
        if (sh.splits == 1) vis_linear_residual(p, old, m0 + q4 * 32, n0 + c * 32, lane);
        tmem_ld32(src + c * 32, r);
        tmem_ld_wait();
        if (c == chunks - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(accfree + 8 * buf);
        }
        if (sh.splits == 1) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          if (n0 + c * 32 < p.N) vis_linear_store(p, v, old, bias + c * 32, stage, m0 + q4 * 32, n0 + c * 32, lane);
        } else if (live) {                                   // [tile][part][column group of four][128 rows][4]
          float4* part = reinterpret_cast<float4*>(p.ws) + ((static_cast<size_t>(tile) * sh.splits + split) * (sh.bn / 4) + (half * (sh.bn / 2) + c * 32) / 4) * 128 + q4 * 32 + lane;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            __stcg(part + j * 128, make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
        }
      }
      if (sh.splits > 1) {
        __threadfence();
        named_bar_sync(1, 256);
        if (abort_s != 0u) break;
        if (te == 0) {
          const bool last = atomicAdd(p.counters + tile, 1u) == static_cast<uint32_t>(sh.splits) - 1u;
          if (last) p.counters[tile] = 0u;
          __threadfence();
          last_s = last ? 1u : 0u;
        }
        named_bar_sync(1, 256);
        const bool last = last_s != 0u;
        named_bar_sync(1, 256);                    // (read by all before the next tile writes it)
        if (last) {
          __threadfence();
          const float4* parts = reinterpret_cast<const float4*>(p.ws) + (static_cast<size_t>(tile) * sh.splits * (sh.bn / 4) + half * (sh.bn / 8)) * 128 + q4 * 32 + lane;
          for (int c = 0; c < chunks; ++c) {
            float v[32];
            VlResidual old;
            vis_linear_residual(p, old, m0 + q4 * 32, n0 + c * 32, lane);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
            for (int sp = 0; sp < sh.splits; ++sp)
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 f = __ldcg(parts + (static_cast<size_t>(sp) * (sh.bn / 4) + c * 8 + j) * 128);
                v[4 * j] += f.x;
                v[4 * j + 1] += f.y;
                v[4 * j + 2] += f.z;
                v[4 * j + 3] += f.w;
              }
            if (n0 + c * 32 < p.N) vis_linear_store(p, v, old, bias + c * 32, stage, m0 + q4 * 32, n0 + c * 32, lane);
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tm, cols);
}

// Tile width and parts of the reduction: the least time of the busiest SM.  A k-block of a tile takes 640, 700, 840 and 780 clocks at 64, 128, 192
// and 256 features (measured at 4096 rows, beside the copies of all other SMs: far from the products' 128 to 512, so wide tiles pay wherever they
// fill the SMs), and a cut reduction about 300 clocks a feature for its way through memory.
static VisLinearShape vis_linear_shape(int M, int N, int K, int sms) {
  constexpr int kBlock[4] = {640, 700, 840, 780};
  const int KB = (K + 63) / 64, tiles_m = (M + 127) / 128;
  VisLinearShape best = {};
  long long cost = 0;
  for (int bn = 64; bn <= 256; bn += 64)
    for (int splits = 1; splits <= 4; ++splits) {
      const int tiles_n = (N + bn - 1) / bn, per = (KB + splits - 1) / splits;
      if ((splits - 1) * per >= KB || (splits > 1 && tiles_m * tiles_n * splits > sms)) continue;
      const long long rounds = (static_cast<long long>(tiles_m) * tiles_n * splits + sms - 1) / sms;
      const long long c = rounds * per * kBlock[bn / 64 - 1] + (splits > 1 ? 300LL * bn : 0);
      if (best.bn == 0 || c < cost) {
        best = {bn, splits, 0, tiles_n, tiles_m * tiles_n};
        cost = c;
      }
    }
  best.stages = min(kVlStages, kVlSmem / (16384 + best.bn * 128));
  return best;
}

static int vl_sms() {
  static int sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  if (sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  return sms[dev];
}

}  // namespace saber

extern "C" int saber_vis_linear_launch(const saber::VisLinearParams* p, cudaStream_t stream) {
  using namespace saber;
  if (p->M <= 0) return 0;
  const int sms = vl_sms();
  if (sms <= 0 || (p->N_pad & 255) || p->N > p->N_pad || p->N <= 0 || p->K <= 0 || (p->ldo & 7) || p->M > p->M_pad || p->epi < 0 || p->epi > 3 || (p->epi == 3 && p->res == nullptr))
    return static_cast<int>(cudaErrorInvalidValue);
  const VisLinearShape s = vis_linear_shape(p->M, p->N, p->K, sms);
  // (a cut reduction has at most one part an SM: the workspace holds a 256-feature tile and a counter, zero between launches, for each)
  if (s.splits > 1 && (p->ws == nullptr || p->counters == nullptr)) return static_cast<int>(cudaErrorInvalidValue);
  static bool ready[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (!ready[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(vis_linear_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kVlSmem + kVlStage + 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    ready[dev] = true;
  }
  const int items = s.tiles * s.splits;
  return static_cast<int>(launch(vis_linear_kernel, dim3(min(items, sms)), dim3(kVlThreads), s.stages * (16384 + s.bn * 128) + kVlStage + 1024, stream, 0, *p, s));
}
