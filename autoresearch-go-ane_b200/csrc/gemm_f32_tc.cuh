// fp32 products on the tensor cores, with the error of fp32 sums.
//
//   * Operands are cut into three bf16 parts, hi + mid + lo, which together are 2^16 times the fp32 value (3 x 8 significand bits,
//     rounded to nearest at each cut).  The factor is for the low bits of small values, which would fall below the last bit of a bf16,
//     2^-133; 2^-149, the last one of an fp32, comes to lie there.  (Without it operands of 2^-115 had errors of 1.1e-6, of 2^-130 3.6e-2.)
//     Six of the nine products of parts are formed; the three that are left out (mid lo, lo mid, lo lo) are below 2^-25 of the product.
//   * The tensor core truncates what it adds to its accumulator, which over a whole contraction would be a bias of several
//     units in the last place.  An accumulator therefore lives for half a k-block, 32 terms: six passes, the small products first,
//     12 MMAs, and only the last two of them at the size of the sum.  Eight warps then add it to the running sums in registers
//     (round to nearest), while the MMAs fill the next of four accumulators.  (With a whole k-block per accumulator sums of terms
//     of one sign were 7.3e-8 too small on average, now 5.1e-8.)
//   * Against float64, relative 2-norm, FMA kernels -> this one: N(0, 1) operands 2048 x 32000 x 288 3.0e-7 -> 0.8e-7, 2048 x 288 x 32000
//     16e-7 -> 4.1e-7, 32000 x 288 x 2048 5.7e-7 -> 1.6e-7; operands from [0, 1) 2048 x 1536 x 288 2.5e-7 -> 0.73e-7, 768 x 768 x 256 0.69e-7
//     both, 1000 x 2304 x 768 2.1e-7 -> 0.9e-7.
//
// A CTA works on 128 x 128 tiles, persistent: warp 0 issues the copies (two stages of 96 KB, the three parts of both
// operands), warp 1 the MMAs (1536 cycles a k-block; the latency and fill of 96 KB behind two stages bound it, about 2250 cycles),
// warps 2 - 9 hold the sums, 64 columns of a row per thread.  SPLIT: a cluster shares a tile along the contraction (products with
// few tiles and a long one, dW and the head's dX): a CTA parks its sums in shared memory, each warp copies every CTA of the cluster the
// columns which that one finishes (bulk copies, counted by the receiver's mbarrier), and what arrives is summed in rank order.
// An operand that is not finite, or not after the factor, makes the sums infinite or NaN (its other parts are NaN), and so does a sum
// above 2^96; such elements are computed again with fp32 FMAs.
#pragma once

#include "gemm_tc.cuh"

namespace ane {

struct F32TcArgs {
  int M, N, K, kp;  // kp: K rounded up to whole k-blocks, the distance between the parts of an operand
  int out, parts;   // 0: store, 1: accumulate; CTAs per tile
  float alpha;
  const float *res1, *s1, *res2, *s2;  // store only
  int ldres;
  float* C;
  int ldc;
  const float *A, *B;  // the fp32 operands
  int lda, ldb;
};

static constexpr int F32TC_THREADS = 64 + 8 * 32;
static constexpr uint32_t F32TC_PART = GEMM_BM * GEMM_BK * 2, F32TC_STAGE = 6 * F32TC_PART;
static constexpr uint32_t F32TC_SMEM = 2 * F32TC_STAGE + 8 * 4096 + 1024;
static_assert(F32TC_SMEM <= GEMM_SMEM_LIMIT, "pipeline does not fit");
static constexpr float F32TC_SCALE = 65536.f, F32TC_UNSCALE = 1.f / (65536.f * 65536.f);  // of an operand, of a product

__device__ __forceinline__ bool f32tc_bad(float v) { return !(fabsf(v) <= 3.402823466e38f); }

// Sums of 32 rows (from m0, a row per lane) and `cols` columns (from n0, up to 32, a multiple of 4), column e of lane r in dword
// 32 e + r of the warp's 4 KB of shared memory at `at`: those whose bit e is set in `wanted` are formed again as fp32 FMAs.  The lanes share
// the contraction of a row and eight columns and stop where all that is wanted of them is NaN, as a sum is from its first NaN term on.
// (One thread per sum, to the end of the contraction, took 37 ms for 2048 x 1536 x 2048 of NaN, 0.10 ms of finite numbers and 0.50 of NaN
// now; by that a tile of K = 32000 took 0.3 s, of the 0.5 s that the MMA warp waits.)
__device__ __forceinline__ void f32tc_park(uint32_t at, int lane, int e, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (uint32_t)(e * 128 + lane * 4)), "f"(v) : "memory");
}
__device__ __forceinline__ float f32tc_parked(uint32_t at, int lane, int e) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at + (uint32_t)(e * 128 + lane * 4)) : "memory");
  return v;
}
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void f32tc_again(const F32TcArgs& a, int m0, int n0, int cols, uint32_t wanted, uint32_t at) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  for (uint32_t rows = __ballot_sync(0xffffffffu, wanted != 0); rows != 0; rows &= rows - 1) {
    const int r = __ffs((int)rows) - 1, m = m0 + r;
    const uint32_t of_row = __shfl_sync(0xffffffffu, wanted, r);
#pragma unroll 1
    for (int c = 0; c < cols; c += 8) {
      const uint32_t want = of_row >> c & 0xffu;
      if (want == 0) continue;
      const bool both = c + 4 < cols;  // the second four columns exist
      float s[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) s[e] = 0.f;
#pragma unroll 1
      for (int k0 = 0, k1 = 128;; k0 = k1, k1 += 1024) {
        const int end = min(k1, a.K);
#pragma unroll 4
        for (int k = k0 + lane; k < end; k += 32) {
          const float x = A_MN ? a.A[(size_t)k * a.lda + m] : a.A[(size_t)m * a.lda + k];
          float y[8];
          if constexpr (B_MN) {
            const float4* b = reinterpret_cast<const float4*>(a.B + (size_t)k * a.ldb + n0 + c);
            *reinterpret_cast<float4*>(y) = b[0];
            *reinterpret_cast<float4*>(y + 4) = b[both ? 1 : 0];
          } else {
            const float* b = a.B + (size_t)(n0 + c) * a.ldb + k;
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = b[(size_t)(e < 4 || both ? e : 0) * a.ldb];
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) s[e] = fmaf(x, y[e], s[e]);
        }
        __syncwarp();
        uint32_t nan = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) nan |= __any_sync(0xffffffffu, s[e] != s[e]) ? 1u << e : 0u;
        if (end == a.K || (want & ~nan) == 0) break;
      }
      float mine = 0.f;  // lane e's column is c + e
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float t = warp_sum(s[e]);
        if (lane == e) mine = t;
      }
      if (lane < 8 && (want >> lane & 1u) != 0) f32tc_park(at, r, c + lane, mine);
    }
  }
  __syncwarp();
}

template <bool A_MN, bool B_MN, bool SPLIT>
__global__ void __launch_bounds__(F32TC_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                   const __grid_constant__ F32TcArgs a, int* status) {
  extern __shared__ uint8_t f32tc_raw[];
  __shared__ __align__(8) uint64_t bar_full[2], bar_empty[2], bar_tfull[4], bar_tempty[4], bar_sums[8];
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_u32(f32tc_raw) + 1023u) & ~1023u, staging = base + 2 * F32TC_STAGE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (!SPLIT && status != nullptr && *reinterpret_cast<volatile int*>(status) != DEV_OK) return;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(smem_u32(&bar_tfull[s]), 1);
      mbar_init(smem_u32(&bar_tempty[s]), 8);
    }
    if constexpr (SPLIT)
      for (int w = 0; w < 8; ++w) {
        mbar_init(smem_u32(&bar_sums[w]), 1);
        mbar_expect_tx(smem_u32(&bar_sums[w]), 32 * 64 * 4);  // a warp's rows and half of the columns, from all parts together
      }
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  pdl_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_wait();

  const int parts = SPLIT ? a.parts : 1, part = SPLIT ? (int)blockIdx.x % parts : 0;
  const int tiles_m = (a.M + 127) / 128, tiles = tiles_m * ((a.N + 127) / 128);
  const int kblocks = a.kp / GEMM_BK, kb0 = kblocks * part / parts, kb1 = kblocks * (part + 1) / parts;
  const int tile0 = SPLIT ? (int)blockIdx.x / parts : (int)blockIdx.x, step = SPLIT ? tiles : (int)gridDim.x;  // SPLIT: one tile per cluster

  if (warp == 0) {
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      for (int tile = tile0; ok && tile < tiles; tile += step) {
        const int m0 = tile % tiles_m * 128, n0 = tile / tiles_m * 128;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it & 1;
          if (!mbar_wait(smem_u32(&bar_empty[s]), ((it >> 1) & 1) ^ 1, status, DEV_MBAR_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t full = smem_u32(&bar_full[s]), sa = base + s * F32TC_STAGE, sb = sa + 3 * F32TC_PART;
          mbar_expect_tx(full, F32TC_STAGE);
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            const int k = p * a.kp + kb * GEMM_BK;
            const uint32_t da = sa + p * F32TC_PART, db = sb + p * F32TC_PART;
            if constexpr (!A_MN) {
              tma_load_2d(da, &tmA, full, k, m0);
            } else {
              tma_load_2d(da, &tmA, full, m0, k);
              tma_load_2d(da + F32TC_PART / 2, &tmA, full, m0 + 64, k);
            }
            if constexpr (!B_MN) {
              tma_load_2d(db, &tmB, full, k, n0);
            } else {
              tma_load_2d(db, &tmB, full, n0, k);
              tma_load_2d(db + F32TC_PART / 2, &tmB, full, n0 + 64, k);
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                                 ((128u >> 3) << 17) | ((128u >> 4) << 24);
      constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};  // lo hi, hi lo, mid mid, mid hi, hi mid, hi hi
      int it = 0;
      bool ok = true;
      for (int tile = tile0; ok && tile < tiles; tile += step) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it & 1;
          if (!mbar_wait(smem_u32(&bar_full[s]), (it >> 1) & 1, status, DEV_MBAR_TIMEOUT_MMA)) {
            ok = false;
            break;
          }
          const uint32_t sa = base + s * F32TC_STAGE, sb = sa + 3 * F32TC_PART;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int buf = (2 * it + h) & 3;
            ok = ok && mbar_wait(smem_u32(&bar_tempty[buf]), ((it >> 1) & 1) ^ 1, status, DEV_MBAR_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int p = 0; p < 6; ++p) {
              const uint32_t da = sa + pa[p] * F32TC_PART, db = sb + pb[p] * F32TC_PART;
#pragma unroll
              for (int k = 2 * h; k < 2 * h + 2; ++k) {
                const uint64_t ad = A_MN ? make_smem_desc(da + k * 2048, 64 * GEMM_BK * 2, 1024) : make_smem_desc(da + k * 32, 16, 1024);
                const uint64_t bd = B_MN ? make_smem_desc(db + k * 2048, 64 * GEMM_BK * 2, 1024) : make_smem_desc(db + k * 32, 16, 1024);
                tc_mma_bf16(tmem + (uint32_t)(buf * 128), ad, bd, idesc, (p > 0 || k > 2 * h) ? 1u : 0u);
              }
            }
            if (h == 1) tc_commit(smem_u32(&bar_empty[s]));
            tc_commit(smem_u32(&bar_tfull[buf]));
          }
          if (!ok) break;
        }
      }
    }
  } else {
    const int g = warp & 3, half = (warp - 2) >> 2;  // rows [32 g, 32 g + 32), columns [64 half, 64 half + 64) of the tile
    const float a1 = a.res1 && a.s1 ? *a.s1 : 1.f, a2 = a.res2 && a.s2 ? *a.s2 : 1.f;
    const uint32_t stage = staging + (uint32_t)(warp - 2) * 4096u;
    int it = 0;
    bool ok = true;
    for (int tile = tile0; ok && tile < tiles; tile += step) {
      const int m = tile % tiles_m * 128 + g * 32 + lane, n_tile = tile / tiles_m * 128;
      float acc[64];
#pragma unroll
      for (int e = 0; e < 64; ++e) acc[e] = 0.f;
      for (int hb = 2 * kb0; hb < 2 * kb1; ++hb, ++it) {  // halves of k-blocks
        const int s = it & 3;
        if (!mbar_wait(smem_u32(&bar_tfull[s]), (it >> 2) & 1, status, DEV_MBAR_TIMEOUT_EPILOGUE)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t at = tmem + ((uint32_t)(g * 32) << 16) + (uint32_t)(s * 128 + half * 64);
        float v[64];
        __syncwarp();
        tmem_ld_32x32(at, v);
        tmem_ld_32x32(at + 32, v + 32);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[s]));
#pragma unroll
        for (int e = 0; e < 64; ++e) acc[e] += v[e];
      }
      if constexpr (!SPLIT) {
        if (!ok) break;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int n0 = n_tile + half * 64 + p * 32;
          if (n0 >= a.N || m - lane >= a.M) break;  // warp-uniform
          bool bad = false;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            acc[32 * p + e] *= F32TC_UNSCALE;
            bad = bad || f32tc_bad(acc[32 * p + e]);
          }
          if (__any_sync(0xffffffffu, bad)) {
            uint32_t wanted = 0;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (m < a.M && n0 + e < a.N && f32tc_bad(acc[32 * p + e])) wanted |= 1u << e;
            if (elect_one()) tma_store_wait_read<0>();
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 32; ++e) f32tc_park(stage, lane, e, acc[32 * p + e]);
            f32tc_again<A_MN, B_MN>(a, m - lane, n0, min(32, a.N - n0), wanted, stage);
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[32 * p + e] = f32tc_parked(stage, lane, e);
            __syncwarp();
          }
          float4 r1[8], r2[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {  // N % 4 == 0
            const bool in = m < a.M && n0 + 4 * q < a.N;
            r1[q] = in && a.res1 ? *reinterpret_cast<const float4*>(a.res1 + (size_t)m * a.ldres + n0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
            r2[q] = in && a.res2 ? *reinterpret_cast<const float4*>(a.res2 + (size_t)m * a.ldres + n0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
          if (elect_one()) tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            float4 v = make_float4(a.alpha * acc[32 * p + 4 * q], a.alpha * acc[32 * p + 4 * q + 1], a.alpha * acc[32 * p + 4 * q + 2],
                                   a.alpha * acc[32 * p + 4 * q + 3]);
            if (a.res1) { v.x += a1 * r1[q].x; v.y += a1 * r1[q].y; v.z += a1 * r1[q].z; v.w += a1 * r1[q].w; }
            if (a.res2) { v.x += a2 * r2[q].x; v.y += a2 * r2[q].y; v.z += a2 * r2[q].z; v.w += a2 * r2[q].w; }
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(stage + (uint32_t)(lane * 128 + ((q ^ (lane & 7)) << 4))), "f"(v.x), "f"(v.y),
                         "f"(v.z), "f"(v.w)
                         : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (a.out != 0) tma_reduce_add_2d(&tmC, stage, n0, m - lane);
            else tma_store_2d(&tmC, stage, n0, m - lane);
            tma_store_commit();
          }
        }
      } else {
        // Parked over the first stage as [column / 4][lane] float4 per warp; every CTA receives its columns of this warp's rows and
        // half over the second stage.  A CTA finishes 64 / parts columns of each half.
        const uint32_t parked = base + (uint32_t)(warp - 2) * 8192u, landed = base + F32TC_STAGE + (uint32_t)(warp - 2) * 8192u;
        const int cols = 64 / parts;
        const uint32_t piece = (uint32_t)cols / 4 * 512u;
#pragma unroll
        for (int q = 0; q < 16; ++q)
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(parked + (uint32_t)q * 512u + (uint32_t)lane * 16u), "f"(acc[4 * q]), "f"(acc[4 * q + 1]),
                       "f"(acc[4 * q + 2]), "f"(acc[4 * q + 3])
                       : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        cluster_sync_all();  // all CTAs are through their k-blocks: the stages are free
        if (lane < parts) {
          const uint32_t to = (uint32_t)((lane + part) % parts);
          bulk_copy_to_cta(map_to_cta(landed + (uint32_t)part * piece, to), parked + to * piece, piece, map_to_cta(smem_u32(&bar_sums[warp - 2]), to));
        }
        __syncwarp();
        // what the sums are added to is requested while they are on their way (32 columns at most)
        const int n_begin = n_tile + half * 64 + part * cols;
        const float* base1 = a.out != 0 ? a.C : a.res1;
        const int ld1 = a.out != 0 ? a.ldc : a.ldres;
        float4 in1[8], in2[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int n = n_begin + 4 * q;
          const bool in = 4 * q < cols && m < a.M && n < a.N;  // N % 4 == 0
          in1[q] = in && base1 ? *reinterpret_cast<const float4*>(base1 + (size_t)m * ld1 + n) : make_float4(0.f, 0.f, 0.f, 0.f);
          in2[q] = in && a.res2 ? *reinterpret_cast<const float4*>(a.res2 + (size_t)m * a.ldres + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        ok = mbar_wait(smem_u32(&bar_sums[warp - 2]), 0u, status, DEV_MBAR_TIMEOUT_EPILOGUE) && ok;
        auto received = [&](int q, float (&s)[4]) {  // in rank order
          s[0] = s[1] = s[2] = s[3] = 0.f;
          for (int p = 0; p < parts; ++p) {
            float4 t;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
                         : "r"(landed + (uint32_t)p * piece + (uint32_t)q * 512u + (uint32_t)lane * 16u) : "memory");
            s[0] += t.x; s[1] += t.y; s[2] += t.z; s[3] += t.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) s[e] *= F32TC_UNSCALE;
        };
        auto finish = [&](int n, const float (&s)[4], const float4& i1, const float4& i2) {
          float4 v = make_float4(a.alpha * s[0], a.alpha * s[1], a.alpha * s[2], a.alpha * s[3]);
          if (base1) { v.x += a1 * i1.x; v.y += a1 * i1.y; v.z += a1 * i1.z; v.w += a1 * i1.w; }
          if (a.res2) { v.x += a2 * i2.x; v.y += a2 * i2.y; v.z += a2 * i2.z; v.w += a2 * i2.w; }
          *reinterpret_cast<float4*>(a.C + (size_t)m * a.ldc + n) = v;
        };
        uint32_t left = 0;  // columns with a sum among their four that is not finite: after the others
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int n = n_begin + 4 * q;
          if (4 * q >= cols || !ok || m >= a.M || n >= a.N) continue;
          float s[4];
          received(q, s);
          if (f32tc_bad(s[0]) || f32tc_bad(s[1]) || f32tc_bad(s[2]) || f32tc_bad(s[3])) left |= 1u << q;
          else finish(n, s, in1[q], in2[q]);
        }
        if (__any_sync(0xffffffffu, left != 0)) {
          uint32_t wanted = 0;
#pragma unroll 1
          for (int q = 0; q < 8; ++q) {
            float s[4];
            if ((left >> q & 1u) == 0) continue;
            received(q, s);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              f32tc_park(stage, lane, 4 * q + e, s[e]);
              if (f32tc_bad(s[e])) wanted |= 1u << (4 * q + e);
            }
          }
          f32tc_again<A_MN, B_MN>(a, m - lane, n_begin, min(cols, a.N - n_begin), wanted, stage);
#pragma unroll 1
          for (int q = 0; q < 8; ++q) {
            const int n = n_begin + 4 * q;
            if ((left >> q & 1u) == 0) continue;
            const float s[4] = {f32tc_parked(stage, lane, 4 * q), f32tc_parked(stage, lane, 4 * q + 1), f32tc_parked(stage, lane, 4 * q + 2),
                                f32tc_parked(stage, lane, 4 * q + 3)};
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            finish(n, s, base1 ? *reinterpret_cast<const float4*>(base1 + (size_t)m * ld1 + n) : zero,
                   a.res2 ? *reinterpret_cast<const float4*>(a.res2 + (size_t)m * a.ldres + n) : zero);
          }
        }
      }
    }
    if constexpr (!SPLIT)
      if (elect_one()) tma_store_wait<0>();
  }
  if constexpr (SPLIT)
    if (warp < 2) {
      __syncwarp();
      cluster_sync_all();
    }
  tc_fence_before();
  __syncthreads();
  if constexpr (SPLIT) cluster_sync_all();  // every CTA has received its sums: this one's copies have been read
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace ane
