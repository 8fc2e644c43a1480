// Causal attention of prompt portions over tiled keys and values, on tcgen05: expanded latents (mla.cu) and
// grouped-query pages (gqa.cu).
//
// A CTA owns 128 query rows of one head and walks the keys its rows can see 128 (two pages) at a time.
//   warp 0     bulk copies: key tiles [k-block of 64][128 keys][128 bytes] and transposed value tiles
//              [page][value row][64 keys], both stored swizzled, two stages each
//   warp 1     one lane issues S = Q K^T into one of two 128-column score buffers, a tile ahead of the softmax,
//              and O += P V with P in tensor memory
//   warps 2-9  softmax, two threads per query row, half of the keys each: scores from tensor memory, running maximum
//              (the halves meet in shared memory), bf16 probabilities back to tensor memory.  O is rescaled only when a row's maximum has grown by more than 2^8 since the
//              factor in use was chosen (the factor cancels in the division at the end).
#include "flash_tc.h"
#include "launch.cuh"
#include "mla_device.cuh"

namespace saber {

constexpr int kTcThreads = 320;
constexpr int kTcKeys = 128;
constexpr float kTcLog2e = 1.4426950408889634f;
constexpr float kTcSlack = 8.f;
constexpr float kTcNone = -1e30f;          // no key seen yet

__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// cap tanh(z s) from 2^(2 z s log2 e): zs is 2 z log2 e.  (Large sums give cap, tiny ones -cap.)
__device__ __forceinline__ float soft_cap(float s, float zs, float cap) { return cap - __fdividef(2.f * cap, 1.f + ex2(s * zs)); }

// tanh(z) = z P(z^2) for |z| <= 0.75 to a relative error of 1e-7: interpolation of tanh(z) / z in the Chebyshev points
// of z^2, in powers of z^2
constexpr float kTanhReach = 0.75f;
constexpr int kTanhTerms = 7;
__constant__ float kTanh[kTanhTerms] = {1.f, -0.33333307505f, 0.13332590461f, -0.05388652161f, 0.02143389918f, -0.00763178663f, 0.00172316108f};

// 32 accumulator columns from c on of a live row into the output's operand.
__device__ __forceinline__ void flash_store(const FlashParams& p, const uint32_t (&r)[32], float inv, const float* g, int m, int k0, int c) {
  if ((p.V & 7) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (c + i * 8 >= p.V) break;
      float y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(r[i * 8 + e]) * inv;
      if (g != nullptr) {
        const float4 ga = *reinterpret_cast<const float4*>(g + c + i * 8), gb = *reinterpret_cast<const float4*>(g + c + i * 8 + 4);
        const float gg[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = y[e] / (1.f + expf(-gg[e]));
      }
      operand_store8(p.out, m, k0 + c + i * 8, y);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (c + i < p.V) {
      const float y = __uint_as_float(r[i]) * inv;
      operand_store1(p.out, m, k0 + c + i, g != nullptr ? y / (1.f + expf(-g[c + i])) : y);
    }
}

// grid (query tiles of the longest possible portion, H, nseq)
__global__ void __launch_bounds__(kTcThreads) flash_tc_kernel(const __grid_constant__ FlashParams p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[16];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t abort_s[4];          // per pair of softmax warps
  __shared__ float half_s[2][2][128];               // [block parity][half of the keys][row]
  const int h = blockIdx.y, j = blockIdx.z;
  const int r0 = p.cu_rows[j], nrows = p.cu_rows[j + 1] - r0;
  const int tiles = (nrows + 127) / 128;
  if (static_cast<int>(blockIdx.x) >= tiles) return;
  const int qt = tiles - 1 - static_cast<int>(blockIdx.x);          // long rows of keys first
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int DK = p.DK, KB = (DK + 63) >> 6, VP = p.VP;
  const int m0 = r0 + qt * 128, rows = min(128, nrows - qt * 128);
  const int pos0 = p.kv_len[j] - nrows + qt * 128;                  // position of the tile's first row
  const int keys = pos0 + rows;
  const int first = first_key(pos0, p.chunk, p.window);             // first key any row of the tile sees
  const int b0 = first / kTcKeys, blocks = (keys + kTcKeys - 1) / kTcKeys - b0;
  const uint32_t q_s = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t kbytes = static_cast<uint32_t>(KB) * 16384u, vbytes = static_cast<uint32_t>(VP) * 256u;
  const uint32_t k_s = q_s + kbytes, v_s = k_s + 2 * kbytes;
  const uint32_t bar = smem_u32(bars);
  const uint32_t kfull = bar, kfree = bar + 16, vfull = bar + 32, vfree = bar + 48, sfull = bar + 64, sfree = bar + 80, pfull = bar + 96,
                 odone = bar + 104, bend = bar + 112;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(kfull + 8 * i, 1);
      mbar_init(kfree + 8 * i, 1);
      mbar_init(vfull + 8 * i, 1);
      mbar_init(vfree + 8 * i, 1);
      mbar_init(sfull + 8 * i, 1);
      mbar_init(sfree + 8 * i, 8);
    }
    for (int i = 0; i < 4; ++i) abort_s[i] = 0u;
    mbar_init(pfull, 8);
    mbar_init(odone, 1);
    mbar_init(bend, 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  // query tile, swizzled; columns past DK and rows past the live ones are zeros
  const __nv_bfloat16* qg = static_cast<const __nv_bfloat16*>(p.q) + (static_cast<size_t>(m0) * p.H + h) * DK;
  for (int r = warp; r < 128; r += 10)
    for (int c = lane; c < KB * 8; c += 32) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < rows && c * 8 < DK) v = *reinterpret_cast<const uint4*>(qg + static_cast<size_t>(r) * p.H * DK + c * 8);
      asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(q_s + (c >> 3) * 16384 + sw128_offset(r, (c & 7) * 16)), "r"(v.x), "r"(v.y),
                   "r"(v.z), "r"(v.w) : "memory");
    }
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_base_s, tm_o = tm + 256, tm_p = tm + 448;

  if (warp == 0) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      const uint8_t* ke = static_cast<const uint8_t*>(p.k);
      const uint8_t* ve = static_cast<const uint8_t*>(p.v);
      const int last = (keys - 1) / 64, g = h / (p.H / p.G);
      int b = 0;
      bool ok = true;
      for (; b < blocks; ++b) {
        const int s = b & 1;
        const uint32_t ph = ((b >> 1) & 1) ^ 1;                     // of the use before this one
        size_t at[2];                                               // (a missing second page: the first again, its keys are masked)
        const int pg = (b0 + b) * 2;
        at[0] = static_cast<size_t>(page_at(p, j, pg)) * p.G + g;
        at[1] = pg + 1 <= last ? static_cast<size_t>(page_at(p, j, pg + 1)) * p.G + g : at[0];
        if (b >= 2 && !mbar_wait(kfree + 8 * s, ph, p.err, kErrWaitEmpty)) { ok = false; break; }
        mbar_arrive_expect_tx(kfull + 8 * s, kbytes);
        for (int kb = 0; kb < KB; ++kb)
          for (int i = 0; i < 2; ++i)
            bulk_g2s(k_s + s * kbytes + kb * 16384 + i * 8192, ke + at[i] * p.k_stride + static_cast<size_t>(kb) * 8192, 8192, kfull + 8 * s);
        if (b >= 2 && !mbar_wait(vfree + 8 * s, ph, p.err, kErrWaitEmpty)) {
          mbar_wait(kfull + 8 * s, (b >> 1) & 1, p.err, kErrWaitDrain);
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(vfull + 8 * s, vbytes);
        for (int i = 0; i < 2; ++i) bulk_g2s(v_s + s * vbytes + i * (vbytes >> 1), ve + at[i] * p.v_stride, vbytes >> 1, vfull + 8 * s);
      }
      if (!ok)                                                      // do not leave while an own copy is in flight
        for (int i = max(0, b - 2); i < b; ++i) {
          mbar_wait(kfull + 8 * (i & 1), (i >> 1) & 1, p.err, kErrWaitDrain);
          mbar_wait(vfull + 8 * (i & 1), (i >> 1) & 1, p.err, kErrWaitDrain);
        }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t id_s = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, 128);
      const uint32_t id_o = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, static_cast<uint32_t>(VP));
      const int steps = DK >> 4;
      auto score = [&](int b) -> bool {                             // S of block b
        const int s = b & 1;
        if (!mbar_wait(kfull + 8 * s, (b >> 1) & 1, p.err, kErrWaitReady)) return false;
        if (b >= 2 && !mbar_wait(sfree + 8 * s, ((b >> 1) & 1) ^ 1, p.err, kErrWaitReady)) return false;
        tc_fence_after_sync();
        for (int t = 0; t < steps; ++t) {
          const uint32_t off = static_cast<uint32_t>(t >> 2) * 16384u + static_cast<uint32_t>(t & 3) * 32u;
          mma_f16_ss(tm + s * 128, make_desc_k128(q_s) + (off >> 4), make_desc_k128(k_s + s * kbytes) + (off >> 4), id_s, t != 0 ? 1u : 0u);
        }
        mma_commit(sfull + 8 * s);
        mma_commit(kfree + 8 * s);
        return true;
      };
      bool ok = score(0);
      for (int b = 0; ok && b < blocks; ++b) {
        if (b + 1 < blocks && !score(b + 1)) { ok = false; break; }
        const int s = b & 1;
        if (!mbar_wait(vfull + 8 * s, (b >> 1) & 1, p.err, kErrWaitReady) || !mbar_wait(pfull, b & 1, p.err, kErrWaitReady)) { ok = false; break; }
        tc_fence_after_sync();
        for (int t = 0; t < 8; ++t) {
          const uint32_t off = static_cast<uint32_t>(t >> 2) * (vbytes >> 1) + static_cast<uint32_t>(t & 3) * 32u;
          mma_bf16_ts(tm_o, tm_p + t * 8, make_desc_k128(v_s + s * vbytes) + (off >> 4), id_o, (b != 0 || t != 0) ? 1u : 0u);
        }
        mma_commit(odone);
        mma_commit(vfree + 8 * s);
      }
      mma_commit(bend);                                             // everything issued has retired before the tensor memory goes back
      mbar_wait(bend, 0, p.err, kErrWaitDrain);
    }
  } else {
    // ---------------------------------------------------------------- softmax
    const int q4 = warp & 3, row = q4 * 32 + lane, half = (warp - 2) >> 2;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const bool capped = p.softcap > 0.f, series = capped && p.bound > 0.f && fabsf(p.scale) * p.bound <= kTanhReach * p.softcap;
    // scores in the base-2 domain: sc times what v holds (1 where the cap already brought them there)
    const float sc = series ? 1.f : capped ? kTcLog2e : p.scale * kTcLog2e, zs = capped ? 2.f * kTcLog2e * p.scale / p.softcap : 0.f;
    f32x2 co[kTanhTerms];
    {
      const float z2 = capped ? (p.scale / p.softcap) * (p.scale / p.softcap) : 0.f;
      float f = p.scale * kTcLog2e;
#pragma unroll
      for (int i = 0; i < kTanhTerms; ++i) {
        co[i] = pack_f2(kTanh[i] * f, kTanh[i] * f);
        f *= z2;
      }
    }
    // (a row may meet blocks ahead of its first key: the maximum starts finite so that differences stay numbers)
    float mx = kTcNone, used = kTcNone, l = 0.f;
    const int low = first_key(pos0 + row, p.chunk, p.window);       // first key of this row
    const int low_last = first_key(pos0 + q4 * 32 + 31, p.chunk, p.window);
    // A wait that runs out ends both warps of a row: the one that gives up arrives at their next meeting without waiting.
    auto give_up = [&]() {
      abort_s[q4] = 1u;
      __threadfence_block();
      named_bar_arrive(1 + q4, 64);
    };
    bool ok = true;
    for (int b = 0; b < blocks; ++b) {
      const int s = b & 1;
      // (waits are decided by the warp as a whole: tensor-memory accesses need all its lanes together)
      ok = __all_sync(0xffffffffu, mbar_wait(sfull + 8 * s, (b >> 1) & 1, p.err, kErrWaitAcc));
      if (!ok) { give_up(); break; }
      tc_fence_after_sync();
      float v[64];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(tm + lane_off + s * 128 + half * 64 + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[c * 32 + i] = __uint_as_float(r[i]);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(sfree + 8 * s);
      if (series) {
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          const f32x2 x = pack_f2(v[i], v[i + 1]), u = mul_f2(x, x);
          f32x2 y = co[kTanhTerms - 1];
#pragma unroll
          for (int t = kTanhTerms - 2; t >= 0; --t) y = fma_f2(y, u, co[t]);
          const float2 f = unpack_f2(mul_f2(x, y));
          v[i] = f.x;
          v[i + 1] = f.y;
        }
      } else if (capped) {
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = soft_cap(v[i], zs, p.softcap);
      }
      const int key0 = (b0 + b) * kTcKeys + half * 64;
      const int vis = pos0 + row - key0, low_v = low - key0;        // last and first visible key of this row inside the half block
      if (key0 + 63 > pos0 + q4 * 32) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i > vis) v[i] = -INFINITY;
      }
      if (low_last > key0) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i < low_v) v[i] = -INFINITY;
      }
      float m4[4] = {mx, mx, mx, mx};
#pragma unroll
      for (int i = 0; i < 64; ++i) m4[i & 3] = fmaxf(m4[i & 3], v[i]);
      mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      half_s[s][half][row] = mx;
      named_bar_sync(1 + q4, 64);
      if (abort_s[q4] != 0u) { ok = false; break; }
      mx = fmaxf(mx, half_s[s][half ^ 1][row]);
      // P and O of the block before are consumed
      ok = __all_sync(0xffffffffu, b == 0 || mbar_wait(odone, (b - 1) & 1, p.err, kErrWaitAcc));
      if (!ok) { give_up(); break; }
      const bool grow = b == 0 || (mx - used) * sc > kTcSlack;
      if (__any_sync(0xffffffffu, grow)) {
        const float f = (grow && b > 0) ? ex2((used - mx) * sc) : 1.f;
        if (grow) used = mx;
        l *= b > 0 ? f : 0.f;
        if (b > 0) {
          tc_fence_after_sync();
          for (int c = half * 32; c < VP; c += 64) {                // (the halves take turns over the columns)
            uint32_t r[32];
            tmem_ld32(tm_o + lane_off + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
            tmem_st32(tm_o + lane_off + c, r);
          }
          tmem_st_wait();
        }
      }
      const float base = used * sc;
      float sum[4] = {};
      {
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float a = ex2(fmaf(v[2 * i], sc, -base)), e = ex2(fmaf(v[2 * i + 1], sc, -base));
          sum[i & 3] += a + e;
          r[i] = pack2(a, e);
        }
        tmem_st32(tm_p + lane_off + half * 32, r);
      }
      tmem_st_wait();
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(pfull);
    }
    if (ok) {
      ok = __all_sync(0xffffffffu, mbar_wait(odone, (blocks - 1) & 1, p.err, kErrWaitAcc));
      if (!ok) give_up();
    }
    if (ok) {
      half_s[blocks & 1][half][row] = l;
      named_bar_sync(1 + q4, 64);
      ok = abort_s[q4] == 0u;
    }
    if (ok) {
      tc_fence_after_sync();
      const int m = m0 + row;
      const bool live = row < rows;
      float den = half_s[blocks & 1][0][row] + half_s[blocks & 1][1][row];
      if (p.sink != nullptr) den += ex2(p.sink[h] * kTcLog2e - used * sc);        // (infinite: the sink takes everything)
      float inv = p.out_scale / den;
      const float* g = p.gate == nullptr ? nullptr : p.gate + static_cast<size_t>(live ? m : m0) * p.ldg + (p.gate_heads ? h : h * p.V);
      if (g != nullptr && p.gate_heads) {
        inv /= 1.f + expf(-g[0]);
        g = nullptr;
      }
      const int k0 = p.out_k0 + h * p.V;
      for (int c = half * 32; c < VP; c += 64) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld32(tm_o + lane_off + c, r);
        tmem_ld_wait();
        if (!live) continue;
        flash_store(p, r, inv, g, m, k0, c);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tm, 512);
}

// ------------------------------------------------------------------------------------ two query tiles per CTA
// Two 128-row query tiles share every key and value tile a CTA fetches: two heads of one key head's group where the group is even,
// else neighbouring row tiles of one head.  One softmax thread owns a query row, a warpgroup a tile; while one tile's scores are in the
// softmax, the tensor cores work on the other's, so that neither waits for the other's latency:
//   MMA order   S0(0) S1(0) | O0 += P0 V, S0(b + 1), O1 += P1 V, S1(b + 1) | ...
// P (bf16) lies over the first half of its own scores: a thread has read its row before it writes.  An MMA-issuing thread's products run in
// order, so the arrival of S(b + 1) also says that O holds block b: the softmax never waits for O.  P goes out in two halves (64 keys, one
// page of values), so that the product of the first starts while the second is still in the exponentials.
// Keys travel in slots of one k-block (128 keys x 64 values), values in slots of a page; as many as fit.
// Bound by the exponentials and the tensor cores in turn (16 exponentials a clock: 2048 clocks for the two tiles' 128 x 128 scores, 1024 for the
// products at 128 columns).  2048 rows behind 2048 tokens: 32 heads of 8 groups at 128 columns 112 us, 920 TFLOP/s (one tile a CTA: 175); 32 heads of
// 192 / 128 columns 134 us (one tile a CTA: 222); 4096 rows that all see each other, 16 heads of 72, 136 us (on `mma.sync`: 302).
// 384 threads: copies, MMA issue and two idle warps, then the two softmax warpgroups.  Launched at 168 registers a thread; the first
// warpgroup hands its share on (56 + 224 + 224 = 3 x 168), because a softmax thread holds a row of 128 scores.
constexpr int kPairThreads = 384;
constexpr int kPairSlots = 8;
constexpr int kPairSmem = 226 * 1024;            // (with the static part at most 227 KB)

struct PairShape {
  int nk, nv;                            // slots of keys, of values
  bool heads;                            // the two tiles are heads of one group
};

__global__ void __launch_bounds__(kPairThreads, 1) flash_pair_kernel(const __grid_constant__ FlashParams p, const PairShape shape) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[4 * kPairSlots + 9];
  __shared__ uint32_t tmem_base_s;
  const int j = blockIdx.z;
  const int r0 = p.cu_rows[j], nrows = p.cu_rows[j + 1] - r0;
  const int tiles = (nrows + 127) / 128, units = shape.heads ? tiles : (tiles + 1) / 2;
  if (static_cast<int>(blockIdx.y) >= units) return;
  const int unit = units - 1 - static_cast<int>(blockIdx.y);        // long rows of keys first
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int DK = p.DK, KB = (DK + 63) >> 6, VP = p.VP;
  const int h0 = static_cast<int>(blockIdx.x) * (shape.heads ? 2 : 1), head_step = shape.heads ? 1 : 0;
  const int qt0 = shape.heads ? unit : unit * 2, qt_step = shape.heads ? 0 : 1;
  const int before = p.kv_len[j] - nrows;                            // tokens ahead of the portion
  const int all = p.kv_len[j];
  auto rows_of = [&](int t) { return max(0, min(128, nrows - (qt0 + t * qt_step) * 128)); };
  const int b0 = p.full ? 0 : first_key(before + qt0 * 128, p.chunk, p.window) / kTcKeys;
  auto blocks_of = [&](int t) {                                      // key blocks of a tile (0: it has no rows)
    const int rows = rows_of(t), keys = p.full ? all : before + (qt0 + t * qt_step) * 128 + rows;
    return rows > 0 ? (keys + kTcKeys - 1) / kTcKeys - b0 : 0;
  };
  const int nb0 = blocks_of(0), nb1 = blocks_of(1), blocks = max(nb0, nb1);
  const uint32_t q_s = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t qbytes = static_cast<uint32_t>(KB) * 16384u, vbytes = static_cast<uint32_t>(VP) * 128u;
  const uint32_t k_s = q_s + 2 * qbytes, v_s = k_s + static_cast<uint32_t>(shape.nk) * 16384u;
  const uint32_t bar = smem_u32(bars);
  const uint32_t kfull = bar, kfree = bar + 8 * kPairSlots, vfull = bar + 16 * kPairSlots, vfree = bar + 24 * kPairSlots,
                 sfull = bar + 32 * kPairSlots, pfull = sfull + 16, odone = pfull + 32, bend = odone + 16;      // pfull: [tile][half]
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4 * kPairSlots + 2; ++i) mbar_init(bar + 8 * i, 1);
    for (int i = 0; i < 4; ++i) mbar_init(pfull + 8 * i, 4);
    for (int i = 0; i < 3; ++i) mbar_init(odone + 8 * i, 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_base_s;                                   // S / P of the tiles at 0 and 128, O at 256 and 384

  if (warp < 4) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
   if (warp == 0) {
    // ---------------------------------------------------------------- copies
    if (lane == 0) {
      const uint8_t* ke = static_cast<const uint8_t*>(p.k);
      const uint8_t* ve = static_cast<const uint8_t*>(p.v);
      const int keys = p.full ? all : before + min(nrows, (qt0 + qt_step + 1) * 128), last = (keys - 1) / 64, g = h0 / (p.H / p.G);
      int ks = 0, vs = 0, nks = 0, nvs = 0;                          // next slots, and fills so far
      uint32_t kph = 1, vph = 1;
      bool ok = true;
      // (page ids are requested a block ahead: an id looked up where it is needed costs its copies a memory round trip)
      const int32_t* table = p.block_table + static_cast<size_t>(j) * p.max_blocks;
      auto entry = [&](int i) { return i <= last && i < p.max_blocks ? table[i] : -1; };
      auto checked = [&](int id) -> size_t {                         // (bounds as in page_at)
        if (id < 0 || id >= p.n_blocks) {
          if (p.err) atomicCAS(p.err, 0u, static_cast<uint32_t>(kErrBadIndex));
          id = 0;
        }
        return static_cast<size_t>(id) * p.G + g;
      };
      int next[2] = {entry(b0 * 2), entry(b0 * 2 + 1)};
      for (int b = 0; ok && b < blocks; ++b) {
        size_t at[2];                                               // (a missing second page: the first again, its keys are masked)
        const int pg = (b0 + b) * 2;
        at[0] = checked(next[0]);
        at[1] = pg + 1 <= last ? checked(next[1]) : at[0];
        next[0] = entry(pg + 2);
        next[1] = entry(pg + 3);
        for (int kb = 0; kb < KB; ++kb) {
          if (nks >= shape.nk && !mbar_wait(kfree + 8 * ks, kph, p.err, kErrWaitEmpty)) { ok = false; break; }
          mbar_arrive_expect_tx(kfull + 8 * ks, 16384);
          for (int i = 0; i < 2; ++i) bulk_g2s(k_s + ks * 16384 + i * 8192, ke + at[i] * p.k_stride + static_cast<size_t>(kb) * 8192, 8192, kfull + 8 * ks);
          ++nks;
          if (++ks == shape.nk) { ks = 0; kph ^= 1; }
        }
        for (int i = 0; ok && i < 2; ++i) {
          if (nvs >= shape.nv && !mbar_wait(vfree + 8 * vs, vph, p.err, kErrWaitEmpty)) { ok = false; break; }
          mbar_arrive_expect_tx(vfull + 8 * vs, vbytes);
          bulk_g2s(v_s + vs * vbytes, ve + at[i] * p.v_stride, vbytes, vfull + 8 * vs);
          ++nvs;
          if (++vs == shape.nv) { vs = 0; vph ^= 1; }
        }
      }
      if (!ok) {                                                    // do not leave while an own copy is in flight
        for (int i = max(0, nks - shape.nk); i < nks; ++i) mbar_wait(kfull + 8 * (i % shape.nk), (i / shape.nk) & 1, p.err, kErrWaitDrain);
        for (int i = max(0, nvs - shape.nv); i < nvs; ++i) mbar_wait(vfull + 8 * (i % shape.nv), (i / shape.nv) & 1, p.err, kErrWaitDrain);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    named_bar_sync(1, 288);                                         // the queries are there
    // (one elected lane, four products unrolled: with the descriptors of a loop's runtime index an issue takes 120 clocks and more, whatever the
    // product's size, so far 45 to 64)
    if (elect_one()) {
      const uint32_t id_s = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, 128);
      const uint32_t id_o = make_idesc(kCFmtF32, kFmtBF16, kFmtBF16, 128, static_cast<uint32_t>(VP));
      const int steps = DK >> 4;
      int ks = 0, vs = 0;                                            // first slots of the block whose scores / values come next
      uint32_t kph = 0, vph = 0;
      auto score = [&](const int t, int b) -> bool {                 // S of block b; behind the second tile its keys are free
        int s = ks;
        uint32_t ph = kph;
        const bool on = b < (t ? nb1 : nb0);
        for (int kb = 0; kb < KB; ++kb) {
          if (on) {
            if (!mbar_wait(kfull + 8 * s, ph, p.err, kErrWaitReady)) return false;
            tc_fence_after_sync();
            const uint64_t qd = make_desc_k128(q_s + t * qbytes + kb * 16384u), kd = make_desc_k128(k_s + s * 16384u);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (kb * 4 + i < steps) mma_f16_ss(tm + t * 128, qd + 2 * i, kd + 2 * i, id_s, (kb | i) != 0 ? 1u : 0u);
          }
          if (t == 1) mma_commit(kfree + 8 * s);
          if (++s == shape.nk) { s = 0; ph ^= 1; }
        }
        if (on) mma_commit(sfull + 8 * t);
        if (t == 1) {
          ks = s;
          kph = ph;
        }
        return true;
      };
      auto values = [&](const int t, int b) -> bool {                // O += P V of block b; behind the second tile its values are free
        int s = vs;
        uint32_t ph = vph;
        const bool on = b < (t ? nb1 : nb0);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (on) {
            if (!mbar_wait(vfull + 8 * s, ph, p.err, kErrWaitReady) || !mbar_wait(pfull + 16 * t + 8 * i, b & 1, p.err, kErrWaitReady)) return false;
            tc_fence_after_sync();
            const uint64_t vd = make_desc_k128(v_s + s * vbytes);
#pragma unroll
            for (int u = 0; u < 4; ++u) mma_bf16_ts(tm + 256 + t * 128, tm + t * 128 + (i * 4 + u) * 8, vd + 2 * u, id_o, (b | i | u) != 0 ? 1u : 0u);
          }
          if (t == 1) mma_commit(vfree + 8 * s);
          if (++s == shape.nv) { s = 0; ph ^= 1; }
        }
        if (on && b == (t ? nb1 : nb0) - 1) mma_commit(odone + 8 * t);
        if (t == 1) {
          vs = s;
          vph = ph;
        }
        return true;
      };
      bool ok = score(0, 0) && score(1, 0);
      for (int b = 0; ok && b < blocks; ++b)
        ok = values(0, b) && (b + 1 >= blocks || score(0, b + 1)) && values(1, b) && (b + 1 >= blocks || score(1, b + 1));
      mma_commit(bend);                                             // everything issued has retired before the tensor memory goes back
      mbar_wait(bend, 0, p.err, kErrWaitDrain);
    }
   }
  } else {
    // ---------------------------------------------------------------- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // query tiles, swizzled, while the first keys are on their way; columns past DK and rows past the live ones are zeros (eight loads of a thread in
    // flight: with a row a warp and step the 22 round trips to memory were most of a short portion's time, 20 us at 308 rows)
    for (int i0 = threadIdx.x - 128; i0 < 256 * KB * 8; i0 += 8 * 256) {
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + u * 256, rr = i / (KB * 8), c = i - rr * KB * 8, t = rr >> 7, r = rr & 127;
        v[u] = make_uint4(0u, 0u, 0u, 0u);
        if (rr < 256 && r < rows_of(t) && c * 8 < DK)
          v[u] = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) + (static_cast<size_t>(r0 + (qt0 + t * qt_step) * 128 + r) * p.H + h0 + t * head_step) * DK + c * 8);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + u * 256, rr = i / (KB * 8), c = i - rr * KB * 8, t = rr >> 7, r = rr & 127;
        if (rr < 256)
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(q_s + t * qbytes + (c >> 3) * 16384 + sw128_offset(r, (c & 7) * 16)), "r"(v[u].x), "r"(v[u].y),
                       "r"(v[u].z), "r"(v[u].w) : "memory");
      }
    }
    fence_proxy_async_smem();
    named_bar_arrive(1, 288);
    const int t = (warp - 4) >> 2, q4 = warp & 3, row = q4 * 32 + lane, h = h0 + t * head_step;
    const int rows = rows_of(t), pos0 = before + (qt0 + t * qt_step) * 128, nb = t ? nb1 : nb0;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16, tm_s = tm + t * 128 + lane_off, tm_o = tm + 256 + t * 128 + lane_off;
    const bool capped = p.softcap > 0.f, series = capped && p.bound > 0.f && fabsf(p.scale) * p.bound <= kTanhReach * p.softcap;
    // scores in the base-2 domain: sc times what v holds (1 where the cap already brought them there)
    const float sc = series ? 1.f : capped ? kTcLog2e : p.scale * kTcLog2e, zs = capped ? 2.f * kTcLog2e * p.scale / p.softcap : 0.f;
    const float z2 = capped ? (p.scale / p.softcap) * (p.scale / p.softcap) : 0.f;
    // (a row may meet blocks ahead of its first key: the maximum starts finite so that differences stay numbers)
    float mx = kTcNone, used = kTcNone, l = 0.f;
    const int seen = p.full ? all - 1 : pos0 + row, seen0 = p.full ? all - 1 : pos0 + q4 * 32;        // last visible key of this row, of the warp's first
    const int low = p.full ? 0 : first_key(pos0 + row, p.chunk, p.window);                              // first key of this row
    const int low_last = p.full ? 0 : first_key(pos0 + q4 * 32 + 31, p.chunk, p.window);
    bool ok = nb > 0;
    for (int b = 0; ok && b < nb; ++b) {
      // (waits are decided by the warp as a whole: tensor-memory accesses need all its lanes together)
      ok = __all_sync(0xffffffffu, mbar_wait(sfull + 8 * t, b & 1, p.err, kErrWaitAcc));
      if (!ok) break;
      tc_fence_after_sync();
      float v[128];
      {
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tm_s + c * 32, r[c]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 128; ++i) v[i] = __uint_as_float(r[i >> 5][i & 31]);
      }
      if (series) {
        f32x2 co[kTanhTerms];
        float f = p.scale * kTcLog2e;
#pragma unroll
        for (int i = 0; i < kTanhTerms; ++i) {
          co[i] = pack_f2(kTanh[i] * f, kTanh[i] * f);
          f *= z2;
        }
#pragma unroll
        for (int i = 0; i < 128; i += 2) {
          const f32x2 x = pack_f2(v[i], v[i + 1]), u = mul_f2(x, x);
          f32x2 y = co[kTanhTerms - 1];
#pragma unroll
          for (int e = kTanhTerms - 2; e >= 0; --e) y = fma_f2(y, u, co[e]);
          const float2 g = unpack_f2(mul_f2(x, y));
          v[i] = g.x;
          v[i + 1] = g.y;
        }
      } else if (capped) {
#pragma unroll
        for (int i = 0; i < 128; ++i) v[i] = soft_cap(v[i], zs, p.softcap);
      }
      const int key0 = (b0 + b) * kTcKeys;
      const int vis = seen - key0, low_v = low - key0;              // last and first visible key of this row inside the block
      if (key0 + 127 > seen0) {
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i > vis) v[i] = -INFINITY;
      }
      if (low_last > key0) {
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i < low_v) v[i] = -INFINITY;
      }
      float m4[4] = {mx, mx, mx, mx};
#pragma unroll
      for (int i = 0; i < 128; ++i) m4[i & 3] = fmaxf(m4[i & 3], v[i]);
      mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      const bool grow = b == 0 || (mx - used) * sc > kTcSlack;
      if (__any_sync(0xffffffffu, grow)) {
        const float f = (grow && b > 0) ? ex2((used - mx) * sc) : 1.f;
        if (grow) used = mx;
        l *= b > 0 ? f : 0.f;
        if (b > 0) {
          for (int c = 0; c < VP; c += 32) {
            uint32_t r[32];
            tmem_ld32(tm_o + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
            tmem_st32(tm_o + c, r);
          }
        }
      }
      const float base = used * sc;
      const f32x2 sc2 = pack_f2(sc, sc), base2 = pack_f2(-base, -base);
      f32x2 sum2[2] = {};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 x = unpack_f2(fma_f2(pack_f2(v[half * 64 + 2 * i], v[half * 64 + 2 * i + 1]), sc2, base2));
          const float a = ex2(x.x), e = ex2(x.y);
          sum2[i & 1] = add_f2(sum2[i & 1], pack_f2(a, e));
          r[i] = pack2(a, e);
        }
        tmem_st32(tm_s + half * 32, r);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(pfull + 16 * t + 8 * half);
      }
      const float2 sa = unpack_f2(add_f2(sum2[0], sum2[1]));
      l += sa.x + sa.y;
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(odone + 8 * t, 0, p.err, kErrWaitAcc));
    if (ok) {
      tc_fence_after_sync();
      const int m = r0 + (qt0 + t * qt_step) * 128 + row;
      const bool live = row < rows;
      float den = l;
      if (p.sink != nullptr) den += ex2(p.sink[h] * kTcLog2e - used * sc);        // (infinite: the sink takes everything)
      float inv = p.out_scale / den;
      const float* g = p.gate == nullptr ? nullptr : p.gate + static_cast<size_t>(live ? m : r0) * p.ldg + (p.gate_heads ? h : h * p.V);
      if (g != nullptr && p.gate_heads) {
        inv /= 1.f + expf(-g[0]);
        g = nullptr;
      }
      const int k0 = p.out_k0 + h * p.V;
      for (int c = 0; c < VP; c += 32) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld32(tm_o + c, r);
        tmem_ld_wait();
        if (live) flash_store(p, r, inv, g, m, k0, c);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tm, 512);
}

// Slots for a shape: the queries stay, then two pages of values and a block's keys at least, then both in turn (values first: a block has
// two pages of them, and all are in use until the second tile is through).
static PairShape pair_shape(const FlashParams& p) {
  const int KB = (p.DK + 63) / 64, group = p.H / p.G;
  PairShape s = {0, 0, (group & 1) == 0};
  int left = kPairSmem - 1024 - 2 * KB * 16384;
  if (p.VP > 128 || KB > kPairSlots || left < KB * 16384 + 2 * p.VP * 128) return s;
  s.nk = KB;
  s.nv = 2;
  left -= KB * 16384 + 2 * p.VP * 128;
  for (bool more = true; more;) {
    more = false;
    if (s.nv < min(kPairSlots, 4) && left >= p.VP * 128) { ++s.nv; left -= p.VP * 128; more = true; }
    if (s.nk < min(kPairSlots, 2 * KB) && left >= 16384) { ++s.nk; left -= 16384; more = true; }
  }
  return s;
}

static int flash_tc_smem(int DK, int VP) { return 3 * ((DK + 63) / 64) * 16384 + 2 * VP * 256 + 1024; }

}  // namespace saber

// VP: the accumulator shares tensor memory with two score buffers (256 columns) and the probabilities (64)
bool saber_flash_tc_ok(int page, int DK, int VP, float scale, float softcap) {
  return (scale > 0.f || softcap > 0.f) && page == 64 && (VP & 31) == 0 && VP <= 192 && (DK & 15) == 0 && saber::flash_tc_smem(DK, VP) <= 224 * 1024;
}

static int flash_allow(const void* kernel, bool (&ready)[64], int smem) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return static_cast<int>(cudaErrorInvalidDevice);
  if (ready[dev]) return 0;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  ready[dev] = e == cudaSuccess;
  return static_cast<int>(e);
}

int saber_flash_tc(const saber::FlashParams* p, cudaStream_t stream) {
  using namespace saber;
  static bool ready[64], ready_pair[64];
  const PairShape s = pair_shape(*p);
  // Two tiles a CTA wherever they fit and there are two: heads of a group, or more than one tile of rows (175 us against 112, above).  One tile of
  // rows of an odd group would leave the second tile empty, and wide values (VP > 128) leave no tensor memory for it.
  if (s.nk > 0 && (s.heads || p->max_rows > 128 || p->full)) {
    const int e = flash_allow(reinterpret_cast<const void*>(flash_pair_kernel), ready_pair, kPairSmem);
    if (e != 0) return e;
    const int smem = 1024 + 2 * ((p->DK + 63) / 64) * 16384 + s.nk * 16384 + s.nv * p->VP * 128;
    const int tiles = (p->max_rows + 127) / 128;
    return static_cast<int>(launch(flash_pair_kernel, dim3(s.heads ? p->H / 2 : p->H, s.heads ? tiles : (tiles + 1) / 2, p->nseq), dim3(kPairThreads), smem, stream, 0, *p, s));
  }
  if (p->full) return static_cast<int>(cudaErrorInvalidValue);
  const int e = flash_allow(reinterpret_cast<const void*>(flash_tc_kernel), ready, 224 * 1024);
  if (e != 0) return e;
  return static_cast<int>(launch(flash_tc_kernel, dim3((p->max_rows + 127) / 128, p->H, p->nseq), dim3(kTcThreads),
                                 flash_tc_smem(p->DK, p->VP), stream, 0, *p));
}
