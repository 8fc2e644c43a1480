// Keys and values of the pages a prompt portion sees, from their latents, on tcgen05: W_uk c and W_uv c in the tile order that flash_tc.cu copies.
//
// A CTA keeps 128 weight rows (of W_uk, then of W_uv) in shared memory for good and walks its share of the page pairs (128 tokens): weights are
// read once per CTA instead of once per pair, and a pair's latents come from L2.  Keys are the product [tokens x weight rows], values the
// transposed one [weight rows x tokens]: both operands are rows of 128 swizzled bytes, so they only change places, and either way a thread of the
// epilogue holds a whole 128-byte row of the result's tiles.
//   warp 0      MMA issue, two accumulators of 128 columns in turn
//   warps 1-4   latents: 16-byte asynchronous copies into a ring of k-blocks, swizzled for their place
//   warps 5-8   epilogue
// The last CTAs of the grid copy the rotated key parts.
// Bound by the stores of the expanded tiles (32 heads x 256 values x 2 bytes a token, 67 MB at 4096 tokens: 20 us there and back).  4096 tokens, 32 heads of
// 128 + 128 values, rank 512: 66 us; on `mma.sync`, weights read once per pair of pages, 216.
#include "launch.cuh"
#include "mla_device.cuh"

namespace saber {

constexpr int kExThreads = 288, kExStages = 4, kExLag = 2, kExCopyCtas = 20;
constexpr uint32_t kExBlock = 16384;                // 128 rows x 64 bf16

// The i-th pair of pages over all sequences of the step.
struct ExPair {
  int page[2];
};
__device__ __forceinline__ int ex_pairs(const MlaParams& p) {
  int n = 0;
  for (int j = 0; j < p.nseq; ++j)
    if (p.cu_rows[j + 1] > p.cu_rows[j]) n += (p.kv_len[j] + 127) / 128;
  return n;
}
__device__ __forceinline__ ExPair ex_pair(const MlaParams& p, int i) {
  int j = 0;
  for (;; ++j) {
    const int n = p.cu_rows[j + 1] > p.cu_rows[j] ? (p.kv_len[j] + 127) / 128 : 0;
    if (i < n) break;
    i -= n;
  }
  ExPair r;
  r.page[0] = page_at(p, j, i * 2);
  r.page[1] = i * 128 + 64 < p.kv_len[j] ? page_at(p, j, i * 2 + 1) : -1;
  return r;
}

__device__ __forceinline__ void ex_copy_rotated(const MlaParams& p, int cta, int ctas) {
  const __nv_bfloat16* cache = static_cast<const __nv_bfloat16*>(p.cache);
  __nv_bfloat16* ke = static_cast<__nv_bfloat16*>(p.k_exp);
  const int LD = p.CP + p.RP, KB = (p.DP + p.RP + 63) >> 6, rot8 = p.RP / 8, pairs = ex_pairs(p);
  for (int i = cta; i < pairs; i += ctas) {
    const ExPair pr = ex_pair(p, i);
    for (int e = threadIdx.x; e < 128 * p.H * rot8; e += kExThreads) {
      const int c = e % rot8, rest = e / rot8, r = rest & 127, h = rest >> 7, pg = pr.page[r >> 6], key = r & 63, d = p.DP + c * 8;
      if (pg < 0) continue;
      const uint4 v = reinterpret_cast<const uint4*>(cache + (static_cast<size_t>(pg) * 64 + key) * LD + p.CP)[c];
      *reinterpret_cast<uint4*>(ke + ((static_cast<size_t>(pg) * p.H + h) * KB + (d >> 6)) * 4096 + key * 64 + (((((d & 63) >> 3) ^ key) & 7) << 3)) = v;
    }
  }
}

// grid (tiles x parts + kExCopyCtas): tile b % tiles, pairs b / tiles, + parts, ...
__global__ void __launch_bounds__(kExThreads, 1) mla_expand_tc_kernel(const __grid_constant__ MlaParams p, const int tiles, const int parts) {
  if (static_cast<int>(blockIdx.x) >= tiles * parts) {
    pdl_wait();
    ex_copy_rotated(p, blockIdx.x - tiles * parts, kExCopyCtas);
    return;
  }
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[2 * kExStages + 5];
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x % tiles, part = blockIdx.x / tiles;
  const int nk = (p.H * p.D + 127) / 128, LD = p.CP + p.RP, KB = (p.CP + 63) / 64;
  const bool isk = tile < nk;
  const int n0 = (isk ? tile : tile - nk) * 128, per_h = isk ? p.D : p.V, N = p.H * per_h;
  const uint32_t w_s = (smem_u32(smem_raw) + 1023u) & ~1023u, a_s = w_s + static_cast<uint32_t>(KB) * kExBlock;
  const uint32_t full = smem_u32(bars), empty = full + 8 * kExStages, accfull = empty + 8 * kExStages, accfree = accfull + 16, bend = accfree + 16;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kExStages; ++s) {
      mbar_init(full + 8 * s, 4);
      mbar_init(empty + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accfull + 8 * i, 1);
      mbar_init(accfree + 8 * i, 4);
    }
    mbar_init(bend, 1);
    mbar_init_fence();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_s), 256);
    tmem_relinquish();
  }
  {                                                  // weights: no kernel writes them
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(isk ? p.w_uk : p.w_uv);
    for (int i = threadIdx.x; i < 128 * KB * 8; i += kExThreads) {
      const int r = i / (KB * 8), ch = i - r * KB * 8, kb = ch >> 3, c = ch & 7, col = ch * 8;
      const bool live = n0 + r < N && col < p.CP;
      cp16(w_s + kb * kExBlock + r * 128 + (((c ^ r) & 7) << 4), live ? w + static_cast<size_t>(n0 + r) * p.CP + col : w, live);
    }
    cp_commit();
    cp_wait<0>();
  }
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_base_s;
  pdl_wait();
  const int pairs = ex_pairs(p), mine = part < pairs ? (pairs - part + parts - 1) / parts : 0;

  if (warp == 0) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, 128);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 0; ok && i < mine; ++i) {
        const int buf = i & 1;
        if (i >= 2 && !mbar_wait(accfree + 8 * buf, ((i >> 1) & 1) ^ 1, p.err, kErrWaitReady)) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait(full + 8 * s, ph, p.err, kErrWaitReady)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t lat = make_desc_k128(a_s + s * kExBlock), wgt = make_desc_k128(w_s + kb * kExBlock);
#pragma unroll
          for (int j = 0; j < 4; ++j) mma_f16_ss(tm + buf * 128, (isk ? lat : wgt) + 2 * j, (isk ? wgt : lat) + 2 * j, idesc, (kb | j) != 0 ? 1u : 0u);
          mma_commit(empty + 8 * s);
          if (++s == kExStages) { s = 0; ph ^= 1u; }
        }
        if (ok) mma_commit(accfull + 8 * buf);
      }
      mma_commit(bend);                              // everything issued has retired before the tensor memory goes back
      mbar_wait(bend, 0, p.err, kErrWaitDrain);
    }
  } else if (warp < 5) {
    // ---------------------------------------------------------------- latents
    const int t = threadIdx.x - 32, c = t & 7, r0 = t >> 3;
    const __nv_bfloat16* cache = static_cast<const __nv_bfloat16*>(p.cache);
    int it = 0, done = 0;
    bool ok = true;
    auto hand_over = [&]() {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * (done % kExStages));
      ++done;
    };
    for (int i = 0; ok && i < mine; ++i) {
      const ExPair pr = ex_pair(p, part + i * parts);
      for (int kb = 0; kb < KB; ++kb, ++it) {
        const int s = it % kExStages;
        if (it >= kExStages) ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * s, ((it / kExStages) & 1) ^ 1, p.err, kErrWaitEmpty));
        if (!ok) break;
        const bool col = kb * 64 + c * 8 < p.CP;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int r = r0 + 16 * u, pg = pr.page[u >> 2];
          const bool live = col && pg >= 0;
          cp16(a_s + s * kExBlock + r * 128 + (((c ^ r) & 7) << 4), live ? cache + (static_cast<size_t>(pg) * 64 + (r & 63)) * LD + kb * 64 + c * 8 : cache, live);
        }
        cp_commit();
        if (it >= kExLag) {
          cp_wait<kExLag>();
          hand_over();
        }
      }
    }
    cp_wait<0>();
    if (ok)
      while (done < it) hand_over();
  } else {
    // ---------------------------------------------------------------- epilogue
    const int row = (warp & 3) * 32 + lane;
    const uint32_t src = tm + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    __nv_bfloat16* ke = static_cast<__nv_bfloat16*>(p.k_exp);
    __nv_bfloat16* ve = static_cast<__nv_bfloat16*>(p.v_exp);
    const int KT = (p.DP + p.RP + 63) >> 6;
    const int n = n0 + row, hv = n / per_h, v = n - hv * per_h;               // of a value row
    for (int i = 0; i < mine; ++i) {
      const int buf = i & 1;
      const ExPair pr = ex_pair(p, part + i * parts);
      // (decided by the warp as a whole: tensor-memory accesses need all its lanes together)
      if (!__all_sync(0xffffffffu, mbar_wait(accfull + 8 * buf, (i >> 1) & 1, p.err, kErrWaitAcc))) break;
      tc_fence_after_sync();
      const int pg = pr.page[row >> 6], key = row & 63;
      int h = n0 / per_h, d = n0 - h * per_h;                                   // of the next eight key columns
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t r[32];
        tmem_ld32(src + buf * 128 + q * 32, r);
        tmem_ld_wait();
        if (q == 3) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(accfree + 8 * buf);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint4 o;
          o.x = pack2(__uint_as_float(r[8 * e]), __uint_as_float(r[8 * e + 1]));
          o.y = pack2(__uint_as_float(r[8 * e + 2]), __uint_as_float(r[8 * e + 3]));
          o.z = pack2(__uint_as_float(r[8 * e + 4]), __uint_as_float(r[8 * e + 5]));
          o.w = pack2(__uint_as_float(r[8 * e + 6]), __uint_as_float(r[8 * e + 7]));
          const int col = q * 32 + e * 8;
          if (isk) {
            if (pg >= 0 && n0 + col < N)
              *reinterpret_cast<uint4*>(ke + ((static_cast<size_t>(pg) * p.H + h) * KT + (d >> 6)) * 4096 + key * 64 + (((((d & 63) >> 3) ^ key) & 7) << 3)) = o;
            d += 8;
            if (d >= p.D) { d = 0; ++h; }
          } else if (n < N && pr.page[col >> 6] >= 0) {
            *reinterpret_cast<uint4*>(ve + ((static_cast<size_t>(pr.page[col >> 6]) * p.H + hv) * p.VP + v) * 64 + (((((col & 63) >> 3) ^ v) & 7) << 3)) = o;
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
}

}  // namespace saber

// Heads of whole groups of eight values, and weights that stay in shared memory beside the ring.
bool saber_mla_expand_tc_ok(const saber::MlaParams* p) { return p->expand == 2 && (p->D & 7) == 0 && p->CP <= 512; }

int saber_mla_expand_tc(const saber::MlaParams* p, cudaStream_t stream) {
  using namespace saber;
  const int KB = (p->CP + 63) / 64, smem = (KB + kExStages) * static_cast<int>(kExBlock) + 1024;
  static bool ready[64];
  static int sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return static_cast<int>(cudaErrorInvalidDevice);
  if (!ready[dev]) {
    cudaError_t e = cudaFuncSetAttribute(mla_expand_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (8 + kExStages) * static_cast<int>(kExBlock) + 1024);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    ready[dev] = true;
  }
  const int tiles = (p->H * p->D + 127) / 128 + (p->H * p->V + 127) / 128;
  const int parts = max(1, (sms[dev] - kExCopyCtas) / tiles);
  return static_cast<int>(launch(mla_expand_tc_kernel, dim3(tiles * parts + kExCopyCtas), dim3(kExThreads), smem, stream, 0, *p, tiles, parts));
}
