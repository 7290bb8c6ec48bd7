// Causal attention, SIMT path: fp32 math on CUDA cores, any head_dim <= 128, GQA-aware.
// It serves the fp32 parity mode and head sizes the tensor-core kernels do not cover.
//
// Forward restates ane/common.go:61-89 (scores * scale, causal mask, softmax, P*V);
// backward restates ane/train_full.go:261-316 with the score scale as an argument
// (the reference hard-codes 1.0 there).
#include "common.cuh"
#include "kernels.h"

namespace ane {

static constexpr int kMaxHdPerLane = 4;  // head_dim <= 128

// ------------------------------------------------------------------------------------------------
// Training attention in fp32 on the FMA units.  A block of 128 threads keeps 32 rows of one head resident in shared
// memory (queries in the forward and dQ kernels, keys in the dK/dV kernel) and streams tiles of 64 rows of the other
// side.  Thread (ty, tx) owns a 4 x 4 piece of every score tile (resident rows 4 ty .., streamed rows tx + 16 j) and, in
// the products with the tile, 4 resident rows x HDP / 16 columns.  All operands stay row-major with a pitch of HDP + 4
// floats, so score operands are read as float4 along the head dimension without bank conflicts, 64 FMAs for eight
// 16-byte reads; probabilities pass through shared memory transposed, [streamed row][resident row], one float4 per
// streamed row.  32 resident rows (not 64 or 128) because the fp32 modes run with few sequences: 2 x 12 heads x 256
// make 192 blocks.  With few blocks an SM the next tile is on its way (cp.async, two buffers) while one is worked on: a block has its SM
// almost to itself then, and waiting for a tile took a third of the time its products do.  us, forward / dQ / dK and dV: 2 x 12 heads of
// 64, seq 256, 34.7 / 83.2 / 125.2 -> 24.4 / 48.6 / 55.2 (a step of one layer); 8 x 6 heads of 48 32.6 / 54.5 / 70.1 -> 24.8 / 39.4 /
// 45.0.  One warp per query with scalar loads and global atomics, which this replaces, took 709 us for the backward of 2 x 12 heads x 256 x 64.
// ------------------------------------------------------------------------------------------------
namespace {

constexpr int kRes = 32, kStr = 64, kSimtThreads = 128;
constexpr int kShortTiles = 4;  // tiles of keys that attention_dq_short_simt_kernel keeps
constexpr size_t kSmemOfSm = 228 * 1024;  // 1 KB of it goes to each block
constexpr int kPPitch = kRes + 4;  // floats of one streamed row of the probability tile

template <int HDP>
struct Simt {
  static constexpr int kPitch = HDP + 4;
  static constexpr int kResFloats = kRes * kPitch, kStrFloats = kStr * kPitch, kProbFloats = kStr * kPPitch;
  static constexpr bool kTwoBuffers = HDP <= 64;  // of streamed tiles, for fp32: two blocks or more fit an SM
  static constexpr size_t fwd_smem(int bufs) { return sizeof(float) * (kResFloats + 2 * bufs * kStrFloats + kProbFloats); }
  static constexpr size_t kDqSmem = sizeof(float) * (2 * kResFloats + 2 * kStrFloats + kProbFloats);
  static constexpr size_t dq_short_smem(int tiles) {  // two buffers of values
    return sizeof(float) * (2 * kResFloats + (tiles + (tiles < 2 ? tiles : 2)) * kStrFloats + kProbFloats);
  }
  static constexpr size_t dkv_smem(int bufs) { return sizeof(float) * (2 * kResFloats + bufs * (2 * kStrFloats + 3 * kStr) + 2 * kProbFloats); }
};

template <typename T>
__device__ __forceinline__ float4 load4(const T* p) {
  if constexpr (sizeof(T) == 4) {
    return *reinterpret_cast<const float4*>(p);
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
}

// ROWS x hd values (row pitch ld) into shared memory as fp32; rows >= valid and columns >= hd become zero.
template <int HDP, int ROWS, typename T>
__device__ __forceinline__ void load_rows(float* dst, const T* src, int ld, int valid, int hd) {
  constexpr int PER = ROWS * (HDP / 4) / kSimtThreads;
  float4 v[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x + i * kSimtThreads, r = e / (HDP / 4), c = (e - r * (HDP / 4)) * 4;
    v[i] = (r < valid && c < hd) ? load4<T>(src + (size_t)r * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x + i * kSimtThreads, r = e / (HDP / 4), c = (e - r * (HDP / 4)) * 4;
    *reinterpret_cast<float4*>(dst + r * Simt<HDP>::kPitch + c) = v[i];
  }
}

// The same without waiting, for fp32 (others arrive at once): to be waited for with tile_wait().
template <int HDP, int ROWS, typename T>
__device__ __forceinline__ void request_rows(float* dst, const T* src, int ld, int valid, int hd) {
  if constexpr (sizeof(T) != 4) {
    load_rows<HDP, ROWS>(dst, src, ld, valid, hd);
  } else {
#pragma unroll
    for (int i = 0; i < ROWS * (HDP / 4) / kSimtThreads; ++i) {
      const int e = threadIdx.x + i * kSimtThreads, r = e / (HDP / 4), c = (e - r * (HDP / 4)) * 4;
      const bool in = r < valid && c < hd;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * Simt<HDP>::kPitch + c)), "l"(in ? src + (size_t)r * ld + c : src), "r"(in ? 16 : 0)
                   : "memory");
    }
  }
}
__device__ __forceinline__ void tile_wait() {  // everything that any thread has requested
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// s[i][j] = <resident row 4 ty + i, streamed row tx + 16 j>
template <int HDP>
__device__ __forceinline__ void scores(float (&s)[4][4], const float* res, const float* str, int ty, int tx) {
  constexpr int P = Simt<HDP>::kPitch;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
  for (int d = 0; d < HDP; d += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(res + (4 * ty + i) * P + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(str + (tx + 16 * j) * P + d);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[i][j] = fmaf(a[i].x, b[j].x, fmaf(a[i].y, b[j].y, fmaf(a[i].z, b[j].z, fmaf(a[i].w, b[j].w, s[i][j]))));
  }
}

// Columns of thread tx: float4 / float2 groups where the width allows, else every 16th.
template <int HDP>
__device__ __forceinline__ int col_of(int tx, int c) {
  if (HDP == 48) return tx + 16 * c;
  if (HDP == 32) return 2 * tx + c;
  if (c < 4) return 4 * tx + c;
  return HDP == 96 ? 64 + 2 * tx + (c - 4) : 64 + 4 * tx + (c - 4);
}
template <int HDP>
__device__ __forceinline__ void load_cols(float (&v)[HDP / 16], const float* row, int tx) {
  if constexpr (HDP == 48) {
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = row[tx + 16 * c];
  } else if constexpr (HDP == 32) {
    const float2 a = *reinterpret_cast<const float2*>(row + 2 * tx);
    v[0] = a.x; v[1] = a.y;
  } else {
    const float4 a = *reinterpret_cast<const float4*>(row + 4 * tx);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    if constexpr (HDP == 96) {
      const float2 b = *reinterpret_cast<const float2*>(row + 64 + 2 * tx);
      v[4] = b.x; v[5] = b.y;
    } else if constexpr (HDP == 128) {
      const float4 b = *reinterpret_cast<const float4*>(row + 64 + 4 * tx);
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
  }
}
// acc[i][c] += sum_n prob[n][4 ty + i] * str[n][col c]
template <int HDP>
__device__ __forceinline__ void accumulate(float (&acc)[4][HDP / 16], const float* prob, const float* str, int ty, int tx) {
#pragma unroll 4
  for (int n = 0; n < kStr; ++n) {
    const float4 p = *reinterpret_cast<const float4*>(prob + n * kPPitch + 4 * ty);
    float v[HDP / 16];
    load_cols<HDP>(v, str + n * Simt<HDP>::kPitch, tx);
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) {
      acc[0][c] = fmaf(p.x, v[c], acc[0][c]);
      acc[1][c] = fmaf(p.y, v[c], acc[1][c]);
      acc[2][c] = fmaf(p.z, v[c], acc[2][c]);
      acc[3][c] = fmaf(p.w, v[c], acc[3][c]);
    }
  }
}
__device__ __forceinline__ void put_probs(float* prob, const float (&s)[4][4], int ty, int tx) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    *reinterpret_cast<float4*>(prob + (tx + 16 * j) * kPPitch + 4 * ty) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
}
__device__ __forceinline__ float row_max(float v) {  // over the 16 threads of a row
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int HDP>
__device__ __forceinline__ void zero(float (&a)[4][HDP / 16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) a[i][c] = 0.f;
}

// Forward: grid (B * H, query tiles), the longest rows first.
template <int HDP, int BUFS, typename T, typename TO>
__global__ void __launch_bounds__(kSimtThreads)
attention_forward_simt_kernel(const T* __restrict__ qkv, TO* __restrict__ out, float* __restrict__ lse, int seq, int H, int KV, int hd, float scale) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float simt_smem[];
  float* Qs = simt_smem;
  float* Kb = Qs + Simt<HDP>::kResFloats;  // buffers of a tile's keys and values
  float* Ps = Kb + 2 * BUFS * Simt<HDP>::kStrFloats;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int b = blockIdx.x / H, h = blockIdx.x - b * H, kvh = h / (H / KV);
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRes;
  const int ld = (H + 2 * KV) * hd;
  const size_t row0 = (size_t)b * seq;
  const T* kb = qkv + row0 * ld + (size_t)(H + kvh) * hd;
  const T* vb = qkv + row0 * ld + (size_t)(H + KV + kvh) * hd;
  auto request = [&](int k0) {
    float* to = Kb + (k0 / kStr & (BUFS - 1)) * 2 * Simt<HDP>::kStrFloats;
    request_rows<HDP, kStr>(to, kb + (size_t)k0 * ld, ld, seq - k0, hd);
    request_rows<HDP, kStr>(to + Simt<HDP>::kStrFloats, vb + (size_t)k0 * ld, ld, seq - k0, hd);
  };
  request_rows<HDP, kRes>(Qs, qkv + (row0 + q0) * ld + (size_t)h * hd, ld, seq - q0, hd);
  if (BUFS == 2) request(0);
  float m[4], l[4], acc[4][HDP / 16];
  zero<HDP>(acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
  const int last = min(q0 + kRes, seq) - 1;
  for (int k0 = 0; k0 <= last; k0 += kStr) {
    if (BUFS == 1) {
      __syncthreads();
      request(k0);
    }
    tile_wait();  // (and everybody has left the buffer that is filled next)
    const float* Ks = Kb + (k0 / kStr & (BUFS - 1)) * 2 * Simt<HDP>::kStrFloats;
    const float* Vs = Ks + Simt<HDP>::kStrFloats;
    if (BUFS == 2 && k0 + kStr <= last) request(k0 + kStr);
    float s[4][4];
    scores<HDP>(s, Qs, Ks, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = q0 + 4 * ty + i;
      float mx = m[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = k0 + tx + 16 * j <= row ? s[i][j] * scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      mx = row_max(mx);  // finite from the first tile on: every row sees key 0
      const float corr = expf(m[i] - mx);
      m[i] = mx;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = expf(s[i][j] - mx);
        sum += s[i][j];
      }
      l[i] = l[i] * corr + sum;  // this thread's part of the sum
#pragma unroll
      for (int c = 0; c < HDP / 16; ++c) acc[i][c] *= corr;
    }
    put_probs(Ps, s, ty, tx);
    __syncthreads();
    accumulate<HDP>(acc, Ps, Vs, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + 4 * ty + i;
    const float sum = row_sum(l[i]);
    if (row >= seq) continue;
    const float inv = 1.0f / sum;
    TO* op = out + (row0 + row) * (size_t)(H * hd) + (size_t)h * hd;
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) {
      const int d = col_of<HDP>(tx, c);
      if (d < hd) op[d] = from_f<TO>(acc[i][c] * inv);
    }
    if (tx == 0 && lse) lse[((size_t)b * H + h) * seq + row] = m[i] + logf(sum);
  }
}

// Backward, first kernel: row statistics for this scale (maximum, 1 / sum, delta = sum_j P dP; the forward's own do not
// serve, its scale may differ) in one sweep over the keys, dQ in a second.
template <int HDP, typename T, typename TD>
__global__ void __launch_bounds__(kSimtThreads)
attention_dq_simt_kernel(const T* __restrict__ qkv, const TD* __restrict__ d_out, float* __restrict__ dqkv, float* __restrict__ stats, int rows, int seq,
                         int H, int KV, int hd, float scale) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float simt_smem[];
  float* Qs = simt_smem;
  float* dOs = Qs + Simt<HDP>::kResFloats;
  float* Ks = dOs + Simt<HDP>::kResFloats;
  float* Vs = Ks + Simt<HDP>::kStrFloats;
  float* Ps = Vs + Simt<HDP>::kStrFloats;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int b = blockIdx.x / H, h = blockIdx.x - b * H, kvh = h / (H / KV);
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRes;
  const int ld = (H + 2 * KV) * hd;
  const size_t row0 = (size_t)b * seq;
  const T* kb = qkv + row0 * ld + (size_t)(H + kvh) * hd;
  const T* vb = qkv + row0 * ld + (size_t)(H + KV + kvh) * hd;
  load_rows<HDP, kRes>(Qs, qkv + (row0 + q0) * ld + (size_t)h * hd, ld, seq - q0, hd);
  load_rows<HDP, kRes>(dOs, d_out + (row0 + q0) * (size_t)(H * hd) + (size_t)h * hd, H * hd, seq - q0, hd);
  const int last = min(q0 + kRes, seq) - 1;
  float m[4], l[4], dl[4], acc[4][HDP / 16];
  zero<HDP>(acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = dl[i] = 0.f;
  }
  float s[4][4], dp[4][4];
  for (int k0 = 0; k0 <= last; k0 += kStr) {
    __syncthreads();
    load_rows<HDP, kStr>(Ks, kb + (size_t)k0 * ld, ld, seq - k0, hd);
    load_rows<HDP, kStr>(Vs, vb + (size_t)k0 * ld, ld, seq - k0, hd);
    __syncthreads();
    scores<HDP>(s, Qs, Ks, ty, tx);
    scores<HDP>(dp, dOs, Vs, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = q0 + 4 * ty + i;
      float mx = m[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = k0 + tx + 16 * j <= row ? s[i][j] * scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      mx = row_max(mx);
      const float corr = expf(m[i] - mx);
      m[i] = mx;
      l[i] *= corr;
      dl[i] *= corr;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = expf(s[i][j] - mx);
        l[i] += p;
        dl[i] += p * dp[i][j];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    l[i] = 1.0f / row_sum(l[i]);
    dl[i] = row_sum(dl[i]) * l[i];
    const int row = q0 + 4 * ty + i;
    if (tx == 0 && row < seq) {
      float* st = stats + ((size_t)b * H + h) * seq + row;
      st[0] = m[i];
      st[(size_t)rows] = l[i];
      st[(size_t)2 * rows] = dl[i];
    }
  }
  for (int k0 = 0; k0 <= last; k0 += kStr) {
    if (last >= kStr) {  // more than one tile: the first sweep ended on another one
      __syncthreads();
      load_rows<HDP, kStr>(Ks, kb + (size_t)k0 * ld, ld, seq - k0, hd);
      load_rows<HDP, kStr>(Vs, vb + (size_t)k0 * ld, ld, seq - k0, hd);
      __syncthreads();
      scores<HDP>(s, Qs, Ks, ty, tx);
      scores<HDP>(dp, dOs, Vs, ty, tx);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = q0 + 4 * ty + i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // one tile: s holds the scaled and masked scores of the first sweep
        const float sc = last >= kStr ? (k0 + tx + 16 * j <= row ? s[i][j] * scale : -INFINITY) : s[i][j];
        const float p = expf(sc - m[i]) * l[i];
        s[i][j] = p * (dp[i][j] - dl[i]) * scale;
      }
    }
    put_probs(Ps, s, ty, tx);
    __syncthreads();
    accumulate<HDP>(acc, Ps, Ks, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + 4 * ty + i;
    if (row >= seq) continue;
    float* op = dqkv + (row0 + row) * ld + (size_t)h * hd;
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) {
      const int d = col_of<HDP>(tx, c);
      if (d < hd) op[d] = acc[i][c];
    }
  }
}

// The first kernel for two to kShortTiles tiles of keys in fp32: scores and dP of the first sweep stay in registers and the keys in
// shared memory, so that the second sweep is one product instead of three.  (Four tiles with one buffer of values and two blocks an SM: 1 %
// slower in a whole update of 2 x 256 tokens.)
template <int HDP>
__global__ void __launch_bounds__(kSimtThreads)
attention_dq_short_simt_kernel(const float* __restrict__ qkv, const float* __restrict__ d_out, float* __restrict__ dqkv, float* __restrict__ stats, int rows,
                               int seq, int H, int KV, int hd, float scale) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float simt_smem[];
  float* Qs = simt_smem;
  float* dOs = Qs + Simt<HDP>::kResFloats;
  float* Kb = dOs + Simt<HDP>::kResFloats;                // all tiles' keys
  const int held = (seq + kStr - 1) / kStr;                // (shared memory for as many: dq_short_smem())
  float* Vb = Kb + held * Simt<HDP>::kStrFloats;          // buffers of values, two where there are tiles for them
  float* Ps = Vb + min(held, 2) * Simt<HDP>::kStrFloats;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int b = blockIdx.x / H, h = blockIdx.x - b * H, kvh = h / (H / KV);
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRes;
  const int ld = (H + 2 * KV) * hd;
  const size_t row0 = (size_t)b * seq;
  const float* kb = qkv + row0 * ld + (size_t)(H + kvh) * hd;
  const float* vb = qkv + row0 * ld + (size_t)(H + KV + kvh) * hd;
  const int last = min(q0 + kRes, seq) - 1, tiles = last / kStr + 1;
  auto request = [&](int t) {
    if (t >= tiles) return;
    request_rows<HDP, kStr>(Kb + t * Simt<HDP>::kStrFloats, kb + (size_t)t * kStr * ld, ld, seq - t * kStr, hd);
    request_rows<HDP, kStr>(Vb + (t & 1) * Simt<HDP>::kStrFloats, vb + (size_t)t * kStr * ld, ld, seq - t * kStr, hd);
  };
  request_rows<HDP, kRes>(Qs, qkv + (row0 + q0) * ld + (size_t)h * hd, ld, seq - q0, hd);
  request_rows<HDP, kRes>(dOs, d_out + (row0 + q0) * (size_t)(H * hd) + (size_t)h * hd, H * hd, seq - q0, hd);
  request(0);
  float m[4], l[4], dl[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = dl[i] = 0.f;
  }
  float s[kShortTiles][4][4], dp[kShortTiles][4][4];
#pragma unroll
  for (int t = 0; t < kShortTiles; ++t) {
    if (t >= tiles) continue;
    tile_wait();
    request(t + 1);
    scores<HDP>(s[t], Qs, Kb + t * Simt<HDP>::kStrFloats, ty, tx);
    scores<HDP>(dp[t], dOs, Vb + (t & 1) * Simt<HDP>::kStrFloats, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = q0 + 4 * ty + i;
      float mx = m[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[t][i][j] = t * kStr + tx + 16 * j <= row ? s[t][i][j] * scale : -INFINITY;
        mx = fmaxf(mx, s[t][i][j]);
      }
      mx = row_max(mx);
      const float corr = expf(m[i] - mx);
      m[i] = mx;
      l[i] *= corr;
      dl[i] *= corr;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = expf(s[t][i][j] - mx);
        l[i] += p;
        dl[i] += p * dp[t][i][j];
      }
    }
  }
  float acc[4][HDP / 16];
  zero<HDP>(acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    l[i] = 1.0f / row_sum(l[i]);
    dl[i] = row_sum(dl[i]) * l[i];
    const int row = q0 + 4 * ty + i;
    if (tx == 0 && row < seq) {
      float* st = stats + ((size_t)b * H + h) * seq + row;
      st[0] = m[i];
      st[(size_t)rows] = l[i];
      st[(size_t)2 * rows] = dl[i];
    }
  }
#pragma unroll
  for (int t = 0; t < kShortTiles; ++t) {
    if (t >= tiles) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = expf(s[t][i][j] - m[i]) * l[i];
        s[t][i][j] = p * (dp[t][i][j] - dl[i]) * scale;
      }
    if (t > 0) __syncthreads();  // the tile before has been read
    put_probs(Ps, s[t], ty, tx);
    __syncthreads();
    accumulate<HDP>(acc, Ps, Kb + t * Simt<HDP>::kStrFloats, ty, tx);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + 4 * ty + i;
    if (row >= seq) continue;
    float* op = dqkv + (row0 + row) * ld + (size_t)h * hd;
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) {
      const int d = col_of<HDP>(tx, c);
      if (d < hd) op[d] = acc[i][c];
    }
  }
}

// Backward, second kernel: dK and dV of 32 keys over the queries of every head that shares them; no atomics.
template <int HDP, int BUFS, typename T, typename TD>
__global__ void __launch_bounds__(kSimtThreads)
attention_dkv_simt_kernel(const T* __restrict__ qkv, const TD* __restrict__ d_out, float* __restrict__ dqkv, const float* __restrict__ stats, int rows,
                          int seq, int H, int KV, int hd, float scale) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float simt_smem[];
  float* Ks = simt_smem;
  float* Vs = Ks + Simt<HDP>::kResFloats;
  float* Qb = Vs + Simt<HDP>::kResFloats;  // buffers of a tile's queries and output gradients
  float* Ps = Qb + 2 * BUFS * Simt<HDP>::kStrFloats;
  float* Ds = Ps + Simt<HDP>::kProbFloats;
  float* sb = Ds + Simt<HDP>::kProbFloats;  // and of maximum, 1 / sum, delta of the 64 queries
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int b = blockIdx.x / KV, kvh = blockIdx.x - b * KV, group = H / KV;
  const int k0 = (int)blockIdx.y * kRes;
  const int ld = (H + 2 * KV) * hd;
  const size_t row0 = (size_t)b * seq;
  request_rows<HDP, kRes>(Ks, qkv + (row0 + k0) * ld + (size_t)(H + kvh) * hd, ld, seq - k0, hd);
  request_rows<HDP, kRes>(Vs, qkv + (row0 + k0) * ld + (size_t)(H + KV + kvh) * hd, ld, seq - k0, hd);
  auto request = [&](int h, int q0, int buf) {
    float* to = Qb + buf * 2 * Simt<HDP>::kStrFloats;
    request_rows<HDP, kStr>(to, qkv + (row0 + q0) * ld + (size_t)h * hd, ld, seq - q0, hd);
    request_rows<HDP, kStr>(to + Simt<HDP>::kStrFloats, d_out + (row0 + q0) * (size_t)(H * hd) + (size_t)h * hd, H * hd, seq - q0, hd);
    for (int i = threadIdx.x; i < 3 * kStr; i += kSimtThreads) {
      const int q = q0 + (i & (kStr - 1));
      sb[buf * 3 * kStr + i] = q < seq ? stats[(size_t)(i / kStr) * rows + ((size_t)b * H + h) * seq + q] : 0.f;
    }
  };
  const int first = k0 / kStr * kStr;
  int buf = 0;
  if (BUFS == 2) request(kvh * group, first, 0);
  float dk[4][HDP / 16], dv[4][HDP / 16];
  zero<HDP>(dk);
  zero<HDP>(dv);
  for (int h = kvh * group; h < (kvh + 1) * group; ++h) {
    for (int q0 = first; q0 < seq; q0 += kStr, buf ^= BUFS - 1) {
      if (BUFS == 1) {
        __syncthreads();
        request(h, q0, 0);
      }
      tile_wait();
      const float* Qs = Qb + buf * 2 * Simt<HDP>::kStrFloats;
      const float* dOs = Qs + Simt<HDP>::kStrFloats;
      const float* st = sb + buf * 3 * kStr;
      if (BUFS == 2) {
        if (q0 + kStr < seq) request(h, q0 + kStr, buf ^ 1);
        else if (h + 1 < (kvh + 1) * group) request(h + 1, first, buf ^ 1);
      }
      float s[4][4], dp[4][4];
      scores<HDP>(s, Ks, Qs, ty, tx);
      scores<HDP>(dp, Vs, dOs, ty, tx);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = tx + 16 * j;
        const float mq = st[q], lq = st[kStr + q], dq = st[2 * kStr + q];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool see = k0 + 4 * ty + i <= q0 + q && q0 + q < seq;
          const float p = see ? expf(s[i][j] * scale - mq) * lq : 0.f;
          s[i][j] = p;
          dp[i][j] = p * (dp[i][j] - dq) * scale;
        }
      }
      put_probs(Ps, s, ty, tx);
      put_probs(Ds, dp, ty, tx);
      __syncthreads();
      accumulate<HDP>(dv, Ps, dOs, ty, tx);
      accumulate<HDP>(dk, Ds, Qs, ty, tx);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = k0 + 4 * ty + i;
    if (row >= seq) continue;
    float* kp = dqkv + (row0 + row) * ld + (size_t)(H + kvh) * hd;
    float* vp = dqkv + (row0 + row) * ld + (size_t)(H + KV + kvh) * hd;
#pragma unroll
    for (int c = 0; c < HDP / 16; ++c) {
      const int d = col_of<HDP>(tx, c);
      if (d < hd) {
        kp[d] = dk[i][c];
        vp[d] = dv[i][c];
      }
    }
  }
}

template <int HDP, int BUFS, typename T, typename TO>
void launch_forward(const T* qkv, TO* out, float* lse, int B, int seq, int H, int KV, int hd, float scale, cudaStream_t s) {
  auto kern = attention_forward_simt_kernel<HDP, BUFS, T, TO>;
  static unsigned long long done = 0;
  smem_opt_in(kern, Simt<HDP>::fwd_smem(BUFS), done);
  launch_pdl(kern, dim3(B * H, (seq + kRes - 1) / kRes), dim3(kSimtThreads), Simt<HDP>::fwd_smem(BUFS), s, qkv, out, lse, seq, H, KV, hd, scale);
}
// Two buffers of streamed tiles, or one and more blocks an SM, which hide one another's loads?  `turns` tiles pass through the longest
// block; `resident` blocks fit the SMs with two buffers.  Step of split precision, six layers of eight heads of 64, us, one / two buffers
// in the forward kernel, and in the one for dK and dV beside two in the forward: seq 256, 384 blocks 2127 / 2093 / 2027, 576 blocks 2511 /
// 2505, 2501 / 2505, 768 blocks 3029 / 3076, 3090 with two for dK and dV alone; seq 128, 384 blocks 1773 / 1760 / 1740, 576 blocks 2062 / 2082,
// 2093.  With one tile there is nothing to request early, but few blocks spread over more SMs: 192 blocks of fp32, four layers,
// 969 / 953 / 936, 512 blocks 1393 / 1421 / 1441.
bool two_buffers(long long blocks, int turns, long long resident) { return blocks <= (turns == 1 ? resident : 148 * (turns < 4 ? 3 : 4)); }

template <int HDP, typename T, typename TO>
void forward_hdp(const T* qkv, TO* out, float* lse, int B, int seq, int H, int KV, int hd, float scale, cudaStream_t s) {
  if constexpr (Simt<HDP>::kTwoBuffers && sizeof(T) == 4) {
    constexpr long long resident = 148 * (kSmemOfSm / (Simt<HDP>::fwd_smem(2) + 1024));
    const long long blocks = (long long)B * H * ((seq + kRes - 1) / kRes);
    if (two_buffers(blocks, (seq + kStr - 1) / kStr, resident)) return launch_forward<HDP, 2>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
  }
  launch_forward<HDP, 1>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
}
template <int HDP, int BUFS, typename T, typename TD>
void launch_dkv(const T* qkv, const TD* d_out, float* dqkv, float* stats, int B, int seq, int H, int KV, int hd, float scale, cudaStream_t s) {
  auto kern = attention_dkv_simt_kernel<HDP, BUFS, T, TD>;
  static unsigned long long done = 0;
  smem_opt_in(kern, Simt<HDP>::dkv_smem(BUFS), done);
  launch_pdl(kern, dim3(B * KV, (seq + kRes - 1) / kRes), dim3(kSimtThreads), Simt<HDP>::dkv_smem(BUFS), s, qkv, d_out, dqkv, stats, B * H * seq, seq, H,
             KV, hd, scale);
}
template <int HDP, typename T, typename TD>
void dkv_hdp(const T* qkv, const TD* d_out, float* dqkv, float* stats, int B, int seq, int H, int KV, int hd, float scale, cudaStream_t s) {
  if constexpr (Simt<HDP>::kTwoBuffers && sizeof(T) == 4) {
    constexpr long long resident = 148 * (kSmemOfSm / (Simt<HDP>::dkv_smem(2) + 1024));
    const long long blocks = (long long)B * KV * ((seq + kRes - 1) / kRes);
    if (two_buffers(blocks, (seq + kStr - 1) / kStr * (H / KV), resident)) return launch_dkv<HDP, 2>(qkv, d_out, dqkv, stats, B, seq, H, KV, hd, scale, s);
  }
  launch_dkv<HDP, 1>(qkv, d_out, dqkv, stats, B, seq, H, KV, hd, scale, s);
}
// dQ of two to four tiles of keys, in fp32: the kernel that keeps everything of its first sweep, with shared memory for the tiles that
// there are.  The same steps, two sweeps / kept: seq 192, 384 blocks 2007 / 1847, 720 blocks 2766 / 2690; head size 48, seq 128, 1176 blocks
// of fp32, 2256 / 2217.  One tile is swept once by the other kernel as well, in less shared memory: 1776 blocks of fp32, 3113 / 3152.  Four
// tiles of head size 64 leave one block an SM, which pays up to four rounds of blocks: seq 256, 384 blocks 2162 / 2027, 448 blocks
// 2303 / 2197, 576 blocks 2556 / 2501, 768 blocks 3029 / 3091.  Two tiles of head size 32 have little to sweep again: 192 blocks of
// fp32, four layers, seq 100, 805 / 792, but seq 128, 960 blocks 1451 / 1496, 1184 blocks 1679 / 1740.
template <int HDP, typename T, typename TD>
void backward_hdp(const T* qkv, const TD* d_out, float* dqkv, float* stats, int B, int seq, int H, int KV, int hd, float scale, cudaStream_t s) {
  const int tiles = (seq + kStr - 1) / kStr, rows = B * H * seq;
  const dim3 grid(B * H, (seq + kRes - 1) / kRes);
  bool kept = false;
  if constexpr (Simt<HDP>::kTwoBuffers && sizeof(T) == 4 && sizeof(TD) == 4) {
    const bool few = (long long)grid.x * grid.y <= 148 * 4;
    kept = tiles > (HDP > 32 || few ? 1 : 2) && tiles <= kShortTiles && (few || 2 * (Simt<HDP>::dq_short_smem(tiles) + 1024) <= kSmemOfSm);
    if (kept) {
      auto kern = attention_dq_short_simt_kernel<HDP>;
      static unsigned long long done = 0;
      smem_opt_in(kern, Simt<HDP>::dq_short_smem(kShortTiles), done);
      launch_pdl(kern, grid, dim3(kSimtThreads), Simt<HDP>::dq_short_smem(tiles), s, qkv, d_out, dqkv, stats, rows, seq, H, KV, hd, scale);
    }
  }
  if (!kept) {
    auto kern = attention_dq_simt_kernel<HDP, T, TD>;
    static unsigned long long done = 0;
    smem_opt_in(kern, Simt<HDP>::kDqSmem, done);
    launch_pdl(kern, grid, dim3(kSimtThreads), Simt<HDP>::kDqSmem, s, qkv, d_out, dqkv, stats, rows, seq, H, KV, hd, scale);
  }
  dkv_hdp<HDP>(qkv, d_out, dqkv, stats, B, seq, H, KV, hd, scale, s);
}

}  // namespace

template <typename T, typename TO>
void attention_forward_simt(const T* qkv, TO* out, float* lse, int B, int seq, int H, int KV, int hd, float scale,
                            cudaStream_t s) {
  if (B <= 0 || seq <= 0) return;
  if (hd <= 32) forward_hdp<32>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
  else if (hd <= 48) forward_hdp<48>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
  else if (hd <= 64) forward_hdp<64>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
  else if (hd <= 96) forward_hdp<96>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
  else forward_hdp<128>(qkv, out, lse, B, seq, H, KV, hd, scale, s);
}
template void attention_forward_simt<float, float>(const float*, float*, float*, int, int, int, int, int, float,
                                                   cudaStream_t);
template void attention_forward_simt<bf16, bf16>(const bf16*, bf16*, float*, int, int, int, int, int, float,
                                                 cudaStream_t);
template void attention_forward_simt<float, bf16>(const float*, bf16*, float*, int, int, int, int, int, float,
                                                  cudaStream_t);

template <typename T, typename TD>
void attention_backward_simt(const T* qkv, const TD* d_out, float* dqkv_f32, float* stats, int B, int seq, int H, int KV, int hd,
                             float scale, cudaStream_t s) {
  if (B <= 0 || seq <= 0) return;
  if (hd <= 32) backward_hdp<32>(qkv, d_out, dqkv_f32, stats, B, seq, H, KV, hd, scale, s);
  else if (hd <= 48) backward_hdp<48>(qkv, d_out, dqkv_f32, stats, B, seq, H, KV, hd, scale, s);
  else if (hd <= 64) backward_hdp<64>(qkv, d_out, dqkv_f32, stats, B, seq, H, KV, hd, scale, s);
  else if (hd <= 96) backward_hdp<96>(qkv, d_out, dqkv_f32, stats, B, seq, H, KV, hd, scale, s);
  else backward_hdp<128>(qkv, d_out, dqkv_f32, stats, B, seq, H, KV, hd, scale, s);
}
template void attention_backward_simt<float, float>(const float*, const float*, float*, float*, int, int, int, int, int, float,
                                                    cudaStream_t);
template void attention_backward_simt<bf16, bf16>(const bf16*, const bf16*, float*, float*, int, int, int, int, int, float,
                                                  cudaStream_t);
template void attention_backward_simt<float, bf16>(const float*, const bf16*, float*, float*, int, int, int, int, int, float,
                                                   cudaStream_t);

// ------------------------------------------------------------------------------------------------
// KV cache for decoding: caches are [B, max_seq, KV*hd].
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void kv_cache_copy_kernel(const T* __restrict__ qkv, T* __restrict__ kcache, T* __restrict__ vcache, int B,
                                     int seq, int max_seq, int pos0, int H, int KV, int hd) {
  const int kvd = KV * hd;
  const int ld = (H + 2 * KV) * hd;
  const long long n = (long long)B * seq * kvd;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % kvd);
    const long long m = i / kvd;
    const int b = (int)(m / seq), t = (int)(m - (long long)b * seq);
    const size_t dst = ((size_t)b * max_seq + pos0 + t) * kvd + c;
    kcache[dst] = qkv[(size_t)m * ld + (size_t)H * hd + c];
    vcache[dst] = qkv[(size_t)m * ld + (size_t)(H + KV) * hd + c];
  }
}
template <typename T>
void kv_cache_fill(const T* qkv, T* kcache, T* vcache, int B, int seq, int max_seq, int H, int KV, int hd,
                   cudaStream_t s) {
  const long long n = (long long)B * seq * KV * hd;
  if (n <= 0) return;
  long long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  kv_cache_copy_kernel<T><<<(unsigned)g, 256, 0, s>>>(qkv, kcache, vcache, B, seq, max_seq, 0, H, KV, hd);
}
template <typename T>
void kv_cache_append(const T* qkv, T* kcache, T* vcache, int B, int max_seq, int pos, int H, int KV, int hd,
                     cudaStream_t s) {
  const long long n = (long long)B * KV * hd;
  if (n <= 0) return;
  kv_cache_copy_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(qkv, kcache, vcache, B, 1, max_seq, pos, H, KV, hd);
}
template void kv_cache_fill<float>(const float*, float*, float*, int, int, int, int, int, int, cudaStream_t);
template void kv_cache_fill<bf16>(const bf16*, bf16*, bf16*, int, int, int, int, int, int, cudaStream_t);
template void kv_cache_append<float>(const float*, float*, float*, int, int, int, int, int, int, cudaStream_t);
template void kv_cache_append<bf16>(const bf16*, bf16*, bf16*, int, int, int, int, int, int, cudaStream_t);

// One warp per (sequence, head): the single query row attends to cache positions 0..pos.
// One block per (sequence, query head); its warps split the cached positions (warp w takes the 32-key
// chunks w, w + kDecWarps, ...), each keeps a running (max, sum, P*V) and the block merges them at the end.
// Key rows are read with 16-byte loads, value rows as one coalesced 128-byte row per key.
static constexpr int kDecWarps = 8;

template <typename T>
__device__ __forceinline__ float dot_row(const float* q, const T* kp, int hd) {
  float dot = 0.f;
  if constexpr (sizeof(T) == 2) {
    for (int d = 0; d < hd; d += 8) {  // hd % 8 == 0 (checked when the engine opens)
      const uint4 u = *reinterpret_cast<const uint4*>(kp + d);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(h2[e]);
        dot += q[d + 2 * e] * f.x + q[d + 2 * e + 1] * f.y;
      }
    }
  } else {
    for (int d = 0; d < hd; d += 4) {
      const float4 f = *reinterpret_cast<const float4*>(kp + d);
      dot += q[d] * f.x + q[d + 1] * f.y + q[d + 2] * f.z + q[d + 3] * f.w;
    }
  }
  return dot;
}

template <typename T>
__global__ void __launch_bounds__(kDecWarps * 32)
attention_decode_simt_kernel(const T* __restrict__ qkv, const T* __restrict__ kcache, const T* __restrict__ vcache,
                             T* __restrict__ out, int B, int max_seq, int pos, int H, int KV, int hd, float scale) {
  extern __shared__ float s_dec[];  // q[hd] | per warp: m, l | per warp: acc[hd]
  float* q = s_dec;
  float* s_m = q + hd;
  float* s_l = s_m + kDecWarps;
  float* s_acc = s_l + kDecWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x / H, h = blockIdx.x - b * H;
  const int kvh = h / (H / KV);
  const int kvd = KV * hd;
  const int ld = (H + 2 * KV) * hd;
  const T* qp = qkv + (size_t)b * ld + (size_t)h * hd;
  for (int d = threadIdx.x; d < hd; d += blockDim.x) q[d] = to_f<T>(qp[d]);
  __syncthreads();
  const T* kbase = kcache + (size_t)b * max_seq * kvd + (size_t)kvh * hd;
  const T* vbase = vcache + (size_t)b * max_seq * kvd + (size_t)kvh * hd;
  float m_run = -INFINITY, l_run = 0.f;
  float acc[kMaxHdPerLane] = {0.f, 0.f, 0.f, 0.f};
  for (int j0 = warp * 32; j0 <= pos; j0 += kDecWarps * 32) {
    const int j = j0 + lane;
    float sc = -INFINITY;
    if (j <= pos) sc = dot_row<T>(q, kbase + (size_t)j * kvd, hd) * scale;
    const float m_new = fmaxf(m_run, warp_max(sc));  // finite: this chunk has at least key j0
    const float corr = __expf(m_run - m_new);
    const float p = (j <= pos) ? __expf(sc - m_new) : 0.f;
    l_run = l_run * corr + warp_sum(p);
#pragma unroll
    for (int c = 0; c < kMaxHdPerLane; ++c) acc[c] *= corr;
    const int lim = min(32, pos - j0 + 1);
    for (int jj = 0; jj < lim; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const T* vp = vbase + (size_t)(j0 + jj) * kvd;
#pragma unroll
      for (int c = 0; c < kMaxHdPerLane; ++c) {
        const int d = lane + 32 * c;
        if (d < hd) acc[c] += pj * to_f<T>(vp[d]);
      }
    }
    m_run = m_new;
  }
  if (lane == 0) {
    s_m[warp] = m_run;
    s_l[warp] = l_run;
  }
#pragma unroll
  for (int c = 0; c < kMaxHdPerLane; ++c) {
    const int d = lane + 32 * c;
    if (d < hd) s_acc[warp * hd + d] = acc[c];
  }
  __syncthreads();
  // merge: warps without any key have m = -inf, l = 0 and drop out
  float m = -INFINITY;
  for (int w = 0; w < kDecWarps; ++w) m = fmaxf(m, s_m[w]);
  float l = 0.f;
  for (int w = 0; w < kDecWarps; ++w) l += s_l[w] * __expf(s_m[w] - m);
  T* op = out + (size_t)b * (H * hd) + (size_t)h * hd;
  for (int d = threadIdx.x; d < hd; d += blockDim.x) {
    float o = 0.f;
    for (int w = 0; w < kDecWarps; ++w) o += s_acc[w * hd + d] * __expf(s_m[w] - m);
    op[d] = from_f<T>(o / l);
  }
}
// head_dim 64, bf16 cache: every lane owns whole keys for BOTH products (its key's score, then p * its value
// row into a private 64-wide accumulator), so a chunk of 32 keys costs sixteen 16-byte loads per lane and
// no shuffles; the lanes' accumulators are summed once at the end.  The query heads that share a KV head
// are handled by separate blocks (their K/V rows then come from L2).
__global__ void __launch_bounds__(kDecWarps * 32, 2)
attention_decode_hd64_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ kcache, const bf16* __restrict__ vcache,
                             bf16* __restrict__ out, int B, int max_seq, int pos, int H, int KV, float scale) {
  constexpr int hd = 64;
  __shared__ float q[hd];
  __shared__ float s_m[kDecWarps], s_l[kDecWarps];
  __shared__ float s_acc[kDecWarps][hd];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x / H, h = blockIdx.x - b * H;
  const int kvh = h / (H / KV);
  const int kvd = KV * hd;
  const int ld = (H + 2 * KV) * hd;
  if (threadIdx.x < hd) q[threadIdx.x] = __bfloat162float(qkv[(size_t)b * ld + (size_t)h * hd + threadIdx.x]);
  __syncthreads();
  const bf16* kbase = kcache + (size_t)b * max_seq * kvd + (size_t)kvh * hd;
  const bf16* vbase = vcache + (size_t)b * max_seq * kvd + (size_t)kvh * hd;
  float m_run = -INFINITY, l_lane = 0.f;
  float acc[hd];
#pragma unroll
  for (int d = 0; d < hd; ++d) acc[d] = 0.f;
  for (int j0 = warp * 32; j0 <= pos; j0 += kDecWarps * 32) {
    const int j = j0 + lane;
    const bool valid = j <= pos;
    float sc = -INFINITY;
    if (valid) {
      uint4 kr[8];
      const uint4* kp = reinterpret_cast<const uint4*>(kbase + (size_t)j * kvd);
#pragma unroll
      for (int c = 0; c < 8; ++c) kr[c] = kp[c];
      float dot = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&kr[c]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(h2[e]);
          dot += q[8 * c + 2 * e] * f.x + q[8 * c + 2 * e + 1] * f.y;
        }
      }
      sc = dot * scale;
    }
    const float m_new = fmaxf(m_run, warp_max(sc));  // finite: this chunk has at least key j0
    const float corr = __expf(m_run - m_new);
    const float p = valid ? __expf(sc - m_new) : 0.f;
    l_lane = l_lane * corr + p;
    if (valid) {
      uint4 vr[8];
      const uint4* vp = reinterpret_cast<const uint4*>(vbase + (size_t)j * kvd);
#pragma unroll
      for (int c = 0; c < 8; ++c) vr[c] = vp[c];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&vr[c]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(h2[e]);
          acc[8 * c + 2 * e] = acc[8 * c + 2 * e] * corr + p * f.x;
          acc[8 * c + 2 * e + 1] = acc[8 * c + 2 * e + 1] * corr + p * f.y;
        }
      }
    } else {
#pragma unroll
      for (int d = 0; d < hd; ++d) acc[d] *= corr;
    }
    m_run = m_new;
  }
  // sum the lanes' partial results (they share m_run), then merge the warps
  const float l_warp = warp_sum(l_lane);
#pragma unroll
  for (int d = 0; d < hd; ++d) {
    const float t = warp_sum(acc[d]);
    if (lane == (d & 31)) s_acc[warp][d] = t;
  }
  if (lane == 0) {
    s_m[warp] = m_run;
    s_l[warp] = l_warp;
  }
  __syncthreads();
  if (threadIdx.x < hd) {
    float m = -INFINITY;
    for (int w = 0; w < kDecWarps; ++w) m = fmaxf(m, s_m[w]);
    float l = 0.f, o = 0.f;
    for (int w = 0; w < kDecWarps; ++w) {
      const float f = __expf(s_m[w] - m);  // warps without any key: exp(-inf) = 0
      l += s_l[w] * f;
      o += s_acc[w][threadIdx.x] * f;
    }
    out[(size_t)b * (H * hd) + (size_t)h * hd + threadIdx.x] = __float2bfloat16_rn(o / l);
  }
}

template <typename T>
void attention_decode_simt(const T* qkv, const T* kcache, const T* vcache, T* out, int B, int max_seq, int pos, int H,
                           int KV, int hd, float scale, cudaStream_t s) {
  const int total = B * H;
  if (total <= 0) return;
  if constexpr (sizeof(T) == 2) {
    if (hd == 64) {
      attention_decode_hd64_kernel<<<total, kDecWarps * 32, 0, s>>>(qkv, kcache, vcache, out, B, max_seq, pos, H, KV, scale);
      return;
    }
  }
  const size_t smem = sizeof(float) * (size_t)(hd + 2 * kDecWarps + kDecWarps * hd);
  attention_decode_simt_kernel<T><<<total, kDecWarps * 32, smem, s>>>(qkv, kcache, vcache, out, B, max_seq, pos, H, KV, hd,
                                                                       scale);
}
template void attention_decode_simt<float>(const float*, const float*, const float*, float*, int, int, int, int, int,
                                           int, float, cudaStream_t);
template void attention_decode_simt<bf16>(const bf16*, const bf16*, const bf16*, bf16*, int, int, int, int, int, int,
                                          float, cudaStream_t);

}  // namespace ane
