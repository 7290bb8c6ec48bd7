// KV-cached generation: all steps after the prefill in ONE persistent cooperative kernel (llama-style architecture,
// bf16 engines).
//
// A decode step is about sixty dependent products with at most 32 rows.  Launched one by one each of them costs the
// fixed latency of a kernel (a 128-row tensor-core tile of the training GEMM takes 10-15 us for 8 KB of useful output),
// although the bytes of a step -- every weight once, keys and values once -- take 35-75 us at the memory's rate.  Here
// one CTA per SM stays resident and walks through the five phases of a layer (q|k|v, attention, Wo, W1|W3, W2).  What
// bounds it is the latency of a phase: how fast one SM's results reach all others, and the chain of instructions
// between reading activations and publishing results.  So:
//   * Weights never change, and the 8 weight rows of a unit are one contiguous piece of 16 K bytes: one thread streams
//     them into a ring of shared-memory slots with bulk copies, as far ahead as the ring reaches, across phases and steps.
//     (Measured with all SMs reading: 30 B/clk per SM through per-lane loads or cp.async, 70 through bulk copies.)
//   * Up to 8 sequences (R8 = 1): results are exchanged as 8-byte words {value, epoch}, written and read with single
//     64-bit accesses.  A reader polls the words it needs; there is no barrier, no fence and no second round trip (a
//     grid barrier with its stores and loads takes 1.8 us on this GPU, a flagged word about 0.6).  A word is not
//     overwritten before everybody has read it: see put_word().
//   * More sequences (R8 = 2, 4): flags would double a traffic that then counts (every SM reads all rows: 98 KB of fp32
//     at 32 x 768), so plain buffers and grid barriers.
//   * All products run through one copy of the code (staging, MMA loop, reduction), so it stays in the instruction cache.
//
// Products: y[b, n] = sum_k x[b, k] W[n, k] with mma.sync m16n8k16 -- the sequences are the A rows (8 of 16 used for
// R8 = 1), 8 weight rows the B columns, so a "unit" of work is 8 weight rows and N / 8 units deal out evenly over the
// SMs.  tcgen05 tiles start at 64 rows of A and would leave most of the tile empty.  Inside a CTA the sixteen warps split
// the contraction in 32-wide chunks (a warp's A fragments then stay in registers for all units of the CTA) and their
// partial sums meet in shared memory.  The order of k inside a chunk is free as long as both operands agree, so every
// lane reads 16 contiguous bytes of a weight row (k = 8 (lane % 4) ..) and uses them as the fragments of two MMAs: no
// ldmatrix.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace ane {
namespace {

constexpr int kWarps = 16, kThreads = kWarps * 32;

// One unit's partial sums of one slice of the contraction: float2 [4 column pairs][rows], pitch free of bank conflicts.
template <int R8>
struct Part {
  static constexpr int kPitch = R8 == 1 ? 12 : 20;
  static constexpr int kTile = 4 * kPitch;  // 8 (R8 = 1) or 16 rows
  static constexpr int kVecs = kTile * (R8 == 4 ? 2 : 1);
};

// `bytes` of global memory into shared memory, counted on the barrier
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Values that other SMs wrote earlier in this kernel: L2 only.  Predicated in one instruction, so that a run of them is
// in flight together.
__device__ __forceinline__ uint4 ld_l2_if(const void* p, bool take) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@p ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"((uint32_t)take) : "memory");
  return v;
}
__device__ __forceinline__ float4 ldf_l2_if(const float* p, bool take) {
  const uint4 v = ld_l2_if(p, take);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u)); }
// sigmoid on the hardware tanh, as in the training forward's epilogue
__device__ __forceinline__ float sigmoid(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}

__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Rows 0-7 only: the accumulators of rows 8-15 are not kept.
__device__ __forceinline__ void mma16816_top(float& c0, float& c1, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  [[maybe_unused]] float x, y;
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, {%7, %8}, {%0, %1, %9, %9};"
               : "+f"(c0), "+f"(c1), "=f"(x), "=f"(y) : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}

// ---- exchange of results between SMs (R8 = 1) -----------------------------------------------------------------------
// Word buffers: x0 (stream after W2), x1 (after Wo), q|k|v, attention out, gate; epoch = step * layers + layer + 1.
// Why a word is never overwritten while someone still needs it: every CTA owns units of q|k|v and of W1|W3 (the grid
// is cut down for that).  x1 of the next layer is written by a CTA that has read all heads' attention outputs, hence all
// q|k|v units of that layer, and each CTA produced its own only after it had read all of x1.  In the same way x0
// follows all gates, hence every CTA's W1|W3 units; gates, attention outputs and q|k|v words follow a complete x1, x0 and
// x0, whose owners had read them.
__device__ __forceinline__ void put_word(uint2* p, uint32_t v, uint32_t epoch) {
  const unsigned long long w = ((unsigned long long)epoch << 32) | v;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
// two neighbouring words: {value, epoch, value, epoch}
__device__ __forceinline__ uint4 get_words(const uint2* p) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}

// Every wait in this kernel is bounded: whoever gives up, or sees in the status word that somebody did, leaves.
struct Wait {
  int* status;
  volatile int* s_abort;
  // called every time a poll failed; true = give up
  __device__ __forceinline__ bool expired(unsigned n, long long& t0) const {
    if ((n & 127u) != 127u) return false;
    const long long t = clock64();
    if (t0 == 0) t0 = t;
    if (t - t0 <= kWaitBudgetCycles && *reinterpret_cast<volatile int*>(status) == DEV_OK) return false;
    atomicCAS(status, DEV_OK, DEV_GRID_TIMEOUT);
    *s_abort = 1;
    return true;
  }
};

// Monotonic arrival counter: barrier number i is complete at i * gridDim.x arrivals.
struct GridBarrier {
  unsigned* count;
  unsigned target;
  Wait wait;
  __device__ __forceinline__ bool sync() {
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("fence.acq_rel.gpu;\n\tred.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      unsigned seen;
      long long t0 = 0;
#pragma unroll 1
      for (unsigned n = 0;; ++n) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
        if ((int)(seen - target) >= 0 || wait.expired(n, t0)) break;
      }
    }
    __syncthreads();
    return *wait.s_abort == 0;
  }
};

// ---- products -------------------------------------------------------------------------------------------------------
enum Kind { kQkv = 0, kWo = 1, kW13 = 2, kW2 = 3, kHead = 4 };
// One product's share of this CTA (in shared memory): `nu` units of 8 weight rows, the first at row `row`, the others in
// alternating steps of inc[0] and inc[1] rows (the grid is a multiple of 4, so W1|W3 blocks keep their phase).
struct Prod {
  size_t off, layer_stride;
  int K, nu, row, inc[2], u0, kind;
  __device__ __forceinline__ int row0(int i) const { return row + (i >> 1) * (inc[0] + inc[1]) + (i & 1) * inc[0]; }
};
__device__ __forceinline__ void make_prod(Prod& d, int kind, size_t off, size_t layer_stride, int K, int n_units) {
  const int g = (int)gridDim.x, b = (int)blockIdx.x;
  d.off = off;
  d.layer_stride = layer_stride;
  d.K = K;
  d.kind = kind;
  d.u0 = 0;
  if (kind == kHead) {  // a contiguous range of the vocabulary
    d.u0 = (int)((long long)n_units * b / g);
    d.nu = (int)((long long)n_units * (b + 1) / g) - d.u0;
    d.row = d.u0 * 8;
    d.inc[0] = d.inc[1] = 8;
  } else if (kind == kW13) {  // W1 and W3 lie in blocks of 32 rows; units 2j and 2j+1 are matching rows of the two
    const int pairs = n_units / 2;
    d.nu = b < pairs ? 2 * ((pairs - b + g - 1) / g) : 0;
    d.row = (b >> 2) * 64 + (b & 3) * 8;
    d.inc[0] = 32;
    d.inc[1] = 16 * g - 32;
  } else {
    d.nu = b < n_units ? (n_units - b + g - 1) / g : 0;
    d.row = b * 8;
    d.inc[0] = d.inc[1] = 8 * g;
  }
}

// The weights of the whole generation in the order they are used, in groups of up to kUnits units of one product, each
// group in one slot of the ring.  One lane of the last warp, which has little to do in the epilogues, issues; a slot is
// free again after the CTA barrier behind its MMAs.
template <int R8>
struct Ring {
  static constexpr int kUnits = R8 == 4 ? 2 : 4;  // per group; even, because W1|W3 units come in pairs
  static constexpr int kSlots = R8 == 4 ? 4 : 3;
};
__device__ __forceinline__ const float* norm_gains(const DecodeArgs& a, int kind, int layer) {
  if (kind == kWo || kind == kW2) return nullptr;
  return a.p + (kind == kHead ? a.off_rms_final : (kind == kQkv ? a.off_rms_att : a.off_rms_ffn) + (size_t)layer * a.rms_stride);
}
template <int R8>
struct Feed {
  uint32_t bar, slot;  // shared-memory addresses of the first barrier and slot
  int slot_bytes, issued, used;
  int step, idx, g0;   // next group
  __device__ __forceinline__ void issue(const DecodeArgs& a, const Prod* prods) {
#pragma unroll 1
    while (issued - used < Ring<R8>::kSlots && step < a.n_new) {
      const int layer = idx >> 2;
      const Prod& p = prods[layer == a.L ? kHead : idx & 3];
      const int n = min(Ring<R8>::kUnits, p.nu - g0);
      if (n > 0) {
        const int at = issued % Ring<R8>::kSlots;
        const uint32_t bytes = (uint32_t)p.K * 16u, b = bar + 8u * at;
        const bf16* w = a.w + p.off + (size_t)layer * p.layer_stride;
        const float* gains = g0 == 0 ? norm_gains(a, p.kind, layer) : nullptr;  // travel with the first group, at the slot's end
        mbar_expect_tx(b, bytes * n + (gains ? a.D * 4u : 0u));
        if (gains) bulk_copy(slot + (uint32_t)((at + 1) * slot_bytes - a.D * 4), gains, a.D * 4u, b);
#pragma unroll 1
        for (int u = 0; u < n; ++u) bulk_copy(slot + (uint32_t)(at * slot_bytes) + bytes * u, w + (size_t)p.row0(g0 + u) * p.K, bytes, b);
        ++issued;
        g0 += n;
      }
      if (g0 >= p.nu) {
        g0 = 0;
        if (++idx > 4 * a.L) {
          idx = 0;
          ++step;
        }
      }
    }
  }
};

// A warp's part of a contraction: chunks [c0, c0 + nc) of 32 columns.
struct Share {
  int K, c0, nc;
};
__device__ __forceinline__ Share make_share(int K) {
  const int warp = threadIdx.x >> 5, chunks = (K + 31) >> 5, per = (chunks + kWarps - 1) / kWarps;
  Share s;
  s.K = K;
  s.c0 = min(warp * per, chunks);
  s.nc = min(per, chunks - s.c0);
  return s;
}

// Where a warp's A fragments come from: normalised rows staged in shared memory, or, for Wo and W2 (no norm, and
// mostly one unit per CTA), straight from the exchanged bf16 rows.
struct Source {
  const uint4* stage;  // nullptr: rows / words
  const bf16* rows;
  const uint2* words;  // R8 = 1: {two values, epoch}
  int B;
  uint32_t epoch;
};
template <int R8>
__device__ __forceinline__ void read_a(uint4 (&f)[4][R8], const Source& s, const Share& w, int first, const Wait& wait) {
  const int lane = threadIdx.x & 31, g = lane >> 2, left = w.nc - first;
  if (s.stage != nullptr) {
    const uint4* st = s.stage + (size_t)(w.c0 + first) * R8 * 32 + lane;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < R8; ++r)
        if (c < left) f[c][r] = st[(c * R8 + r) * 32];
    return;
  }
  const int k = (w.c0 + first) * 32 + (lane & 3) * 8;
  if constexpr (R8 == 1) {
    const uint2* p = s.words + ((size_t)(g < s.B ? g : 0) * w.K + k) / 2;
    long long t0 = 0;
#pragma unroll 1
    for (unsigned n = 0;; ++n) {
      bool ok = true;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint4 x = make_uint4(0, s.epoch, 0, s.epoch), y = x;
        if (c < left && k + c * 32 < w.K && g < s.B) {
          x = get_words(p + c * 16);
          y = get_words(p + c * 16 + 2);
        }
        ok = ok && x.y == s.epoch && x.w == s.epoch && y.y == s.epoch && y.w == s.epoch;
        f[c][0] = make_uint4(x.x, x.z, y.x, y.z);
      }
      if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) return;
    }
  } else {
#pragma unroll
    for (int r = 0; r < R8; ++r) {
      const bool live = r * 8 + g < s.B;
      const bf16* p = s.rows + (size_t)(live ? r * 8 + g : 0) * w.K + k;
#pragma unroll
      for (int c = 0; c < 4; ++c) f[c][r] = ld_l2_if(p + c * 32, live && c < left && k + c * 32 < w.K);
    }
  }
}

// Partial sums of the n units in a slot (rows of K bf16): this warp's chunks.
template <int R8>
__device__ __forceinline__ void run_units(const Share& w, int n, const uint8_t* slot, float2* part, const Source& src, uint4 (&a)[4][R8], bool read, const Wait& wait) {
  constexpr int T = (R8 + 1) / 2;
  using P = Part<R8>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* d = part + (size_t)warp * P::kVecs + (lane & 3) * P::kPitch + (lane >> 2);
  const int k0 = w.c0 * 32 + (lane & 3) * 8;
  const uint4* wp = reinterpret_cast<const uint4*>(slot) + ((lane >> 2) * w.K + k0) / 8;
  float acc[T][4] = {};
#pragma unroll 1
  for (; n > 0; --n) {
#pragma unroll 1
    for (int blk = 0; blk == 0 || blk < w.nc; blk += 4) {
      if (read) read_a<R8>(a, src, w, blk, wait);
      read = w.nc > 4;  // four chunks or fewer: the same fragments for every unit
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (blk + c < w.nc) {
          uint4 b = make_uint4(0, 0, 0, 0);
          if (k0 + (blk + c) * 32 < w.K) b = wp[(blk + c) * 4];
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const uint4 lo = a[c][2 * t], hi = R8 > 1 ? a[c][R8 > 1 ? 2 * t + 1 : 0] : make_uint4(0, 0, 0, 0);
            if constexpr (R8 == 1) {
              mma16816_top(acc[t][0], acc[t][1], lo.x, lo.y, b.x, b.y);
              mma16816_top(acc[t][0], acc[t][1], lo.z, lo.w, b.z, b.w);
            } else {
              mma16816(acc[t], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
              mma16816(acc[t], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
            }
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
      d[t * P::kTile] = make_float2(acc[t][0], acc[t][1]);
      if (R8 > 1) d[t * P::kTile + 8] = make_float2(acc[t][2], acc[t][3]);
      acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    }
    d += kWarps * P::kVecs;
    wp += w.K;
  }
}

// Sum over the warps of column pair (2c, 2c + 1) of row b.
template <int R8>
__device__ __forceinline__ float2 pair_sum(const float2* part, int unit, int b, int c) {
  using P = Part<R8>;
  const float2* d = part + (size_t)unit * kWarps * P::kVecs + (b >> 4) * P::kTile + c * P::kPitch + (b & 15);
  float2 s = make_float2(0.f, 0.f), t = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kWarps; i += 2) {
    const float2 u = d[i * P::kVecs], v = d[(i + 1) * P::kVecs];
    s.x += u.x;
    s.y += u.y;
    t.x += v.x;
    t.y += v.y;
  }
  return make_float2(s.x + t.x, s.y + t.y);
}

// ---- activations into A fragments -------------------------------------------------------------------------------------
// stage[chunk][8-row group][lane]: byte offset of element k of row r.  Rows past the batch stay zero from the start.
template <int R8>
__device__ __forceinline__ int frag_at(int r, int k) {
  return ((((k >> 5) * R8 + (r >> 3)) * 32 + (r & 7) * 4 + ((k & 31) >> 3)) << 4) + (k & 7) * 2;
}

// Which rows a warp normalises: up to 8 sequences share the warps (16 / B per row), more take a warp each, 17 and more
// two rows a warp.
struct RowShare {
  int row, sub, per_row;
};
// Normalised rows, bf16(x * rms^-1 * gain), rounded like the training forward's.  row(r) = plain fp32 values; words:
// {value, epoch} pairs instead (R8 = 1).  A warp's part of a row stays in registers between the sum of squares and the
// conversion for dim <= 768; wider rows go through in segments and are read twice.  gains: the norm's weights in
// shared memory.
template <int R8, class Row>
__device__ __forceinline__ void stage_norm(int K, int B, Row row, const uint2* words, uint32_t epoch, const float* gains, uint8_t* stage,
                                           float* s_sq, const RowShare& sh, const Wait& wait) {
  constexpr int V = R8 == 1 ? 3 : 6;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = sh.per_row * 128, seg = stride * V, nseg = (K + seg - 1) / seg;
#pragma unroll 1
  for (int r = sh.row; r < (R8 == 4 ? B : 16); r += 16) {
    const bool has = r < B;
    const float* px = row(has ? r : 0);
    const uint2* pw = words + (size_t)(has ? r : 0) * K;
    float sq = 0.f, rms = 0.f;
#pragma unroll 1
    for (int it = 0; it < (nseg == 1 ? 1 : 2 * nseg); ++it) {
      const int k0 = (it < nseg ? it : it - nseg) * seg + (sh.sub * 32 + lane) * 4;
      float4 x[V];
#pragma unroll
      for (int i = 0; i < V; ++i) x[i] = ldf_l2_if(px + k0 + i * stride, has && k0 + i * stride < K && (R8 > 1 || words == nullptr));
      if (R8 == 1 && words != nullptr) {
        long long t0 = 0;
#pragma unroll 1
        for (unsigned n = 0;; ++n) {
          bool ok = true;
#pragma unroll
          for (int i = 0; i < V; ++i) {
            if (!has || k0 + i * stride >= K) continue;
            const uint4 a = get_words(pw + k0 + i * stride), b = get_words(pw + k0 + i * stride + 2);
            ok = ok && a.y == epoch && a.w == epoch && b.y == epoch && b.w == epoch;
            x[i] = make_float4(__uint_as_float(a.x), __uint_as_float(a.z), __uint_as_float(b.x), __uint_as_float(b.z));
          }
          if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
        }
      }
      if (it < nseg) {
#pragma unroll
        for (int i = 0; i < V; ++i) sq += (x[i].x * x[i].x + x[i].y * x[i].y) + (x[i].z * x[i].z + x[i].w * x[i].w);
      }
      if (it == nseg - 1) {
        sq = warp_sum(sq);
        if (R8 == 1) {  // the row's other warps
          if (lane == 0) s_sq[warp] = sq;
          __syncthreads();
          sq = 0.f;
#pragma unroll 1
          for (int i = 0; i < sh.per_row; ++i) sq += s_sq[warp - sh.sub + i];
        }
        rms = 1.0f / sqrtf(sq / (float)K + 1e-5f);
      }
      if (it >= nseg || nseg == 1) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
          if (!has || k0 + i * stride >= K) continue;
          const float4 g = *reinterpret_cast<const float4*>(gains + k0 + i * stride);
          *reinterpret_cast<uint2*>(stage + frag_at<R8>(r, k0 + i * stride)) =
              make_uint2(pack2(x[i].x * rms * g.x, x[i].y * rms * g.y), pack2(x[i].z * rms * g.z, x[i].w * rms * g.w));
        }
      }
    }
  }
}

// ---- attention ------------------------------------------------------------------------------------------------------
// One new token per sequence over cache positions 0..pos.  A work item is one sequence and the (up to 8) query heads
// of one KV head, which are the rows of the MMAs; every warp takes 16 keys at a time and keeps a running maximum, sum and
// P*V, merged at the end.  No operand is transposed or staged:
//   scores  B[k = dim, n = key]: lane (g, c) reads 16 bytes of key g at dims 8c.. and 32 + 8c.., two MMAs each (the
//           order of k is free as long as q is read the same way);
//   P * V   B[k = key, n]: lane (g, c) reads dims 8g.. of keys 2c, 2c + 1, 2c + 8, 2c + 9; MMA j takes element j of each, so
//           its column n stands for dim 8n + j.  P enters as bf16 hi + lo, two MMAs, so that it keeps 16 bits.
// hd <= 64 is one panel of 64 dims (what lies past hd reads as zero), up to 128 two.  With flagged words (R8 = 1) q and the
// new key and value come from the words, the older ones from the cache.
template <int R8, int PANELS>
__device__ __forceinline__ void attention_phase(const DecodeArgs& a, const bf16* kc, const bf16* vc, int pos, float* sm, uint32_t epoch, const Wait& wait) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int kvd = a.KV * a.hd, qd = a.H * a.hd, rep = a.H / a.KV, G = a.group, hgroups = a.H / G;
  const float sc = 1.4426950408889634f / sqrtf((float)a.hd);  // scores in the log2 domain
#pragma unroll 1
  for (int item = blockIdx.x; item < a.B * hgroups; item += gridDim.x) {
    const int b = item / hgroups, h0 = (item - b * hgroups) * G, kvh = h0 / rep;
    const bf16* kb = kc + (size_t)b * a.S * kvd + (size_t)kvh * a.hd;
    const bf16* vb = vc + (size_t)b * a.S * kvd + (size_t)kvh * a.hd;
    const uint2* wk = nullptr;  // words of the new key
    // 16 bytes of a key's or value's dims d..d+7 from the cache (R8 = 1: all but the newest, which put_new() adds).  The
    // registers of a tile are requested again as soon as its MMAs have read them: keys load under the softmax and P * V,
    // values under the next scores; the first tiles (the cache does not depend on q) before q is there.
    const int cached = R8 == 1 ? pos : pos + 1;
    uint4 kr[2][2 * PANELS], vr[4][PANELS];
    auto fetch = [&](const bf16* base, int j, int d) { return ld_l2_if(base + (size_t)j * kvd + d, d < a.hd && j < cached); };
    auto load_k = [&](int j0) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int i = 0; i < 2 * PANELS; ++i) kr[t][i] = fetch(kb, j0 + t * 8 + g, i * 32 + c * 8);
    };
    auto load_v = [&](int j0) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int p = 0; p < PANELS; ++p) vr[t][p] = fetch(vb, j0 + 2 * c + (t & 1) + (t >> 1) * 8, p * 64 + g * 8);
    };
    load_k(warp * 16);
    load_v(warp * 16);
    uint4 q[PANELS][2];
    if constexpr (R8 == 1) {
      const uint2* row = a.w_qkv + (size_t)b * ((qd + 2 * kvd) / 2);
      wk = row + (qd + kvh * a.hd) / 2;
      // every word of this item: q rows, key and value (the last two are read again below, from L2 as well)
      long long t0 = 0;
#pragma unroll 1
      for (unsigned n = 0;; ++n) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 2 * PANELS; ++i) {
          const int d = i * 32 + c * 8;
          q[i >> 1][i & 1] = make_uint4(0, 0, 0, 0);
          if (d < a.hd) {
            const uint4 k0 = get_words(wk + d / 2), k1 = get_words(wk + d / 2 + 2), v0 = get_words(wk + (kvd + d) / 2), v1 = get_words(wk + (kvd + d) / 2 + 2);
            ok = ok && k0.y == epoch && k0.w == epoch && k1.y == epoch && k1.w == epoch && v0.y == epoch && v0.w == epoch && v1.y == epoch && v1.w == epoch;
            if (g < G) {
              const uint2* p = row + ((h0 + g) * a.hd + d) / 2;
              const uint4 x = get_words(p), y = get_words(p + 2);
              ok = ok && x.y == epoch && x.w == epoch && y.y == epoch && y.w == epoch;
              q[i >> 1][i & 1] = make_uint4(x.x, x.z, y.x, y.z);
            }
          }
        }
        if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 2 * PANELS; ++i) {
        const int d = i * 32 + c * 8;
        q[i >> 1][i & 1] = ld_l2_if(a.q + (size_t)b * qd + (size_t)(h0 + g) * a.hd + d, g < G && d < a.hd);
      }
    }
    auto put_new = [&](uint4& v, int off, int j, int d) {
      if (R8 == 1 && j == pos && d < a.hd) {
        const uint4 x = get_words(wk + (off + d) / 2), y = get_words(wk + (off + d) / 2 + 2);
        v = make_uint4(x.x, x.z, y.x, y.z);
      }
    };
    float m = -INFINITY, l = 0.f, acc[PANELS][8][2] = {};
#pragma unroll 1
    for (int j0 = warp * 16; j0 <= pos; j0 += kWarps * 16) {
      if (R8 == 1 && j0 + 16 > pos) {  // this warp holds the newest key
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int i = 0; i < 2 * PANELS; ++i) put_new(kr[t][i], 0, j0 + t * 8 + g, i * 32 + c * 8);
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int p = 0; p < PANELS; ++p) put_new(vr[t][p], kvd, j0 + 2 * c + (t & 1) + (t >> 1) * 8, p * 64 + g * 8);
      }
      float s[2][2] = {}, mn = m;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int i = 0; i < 2 * PANELS; ++i) {
          const uint4 k = kr[t][i], x = q[i >> 1][i & 1];
          mma16816_top(s[t][0], s[t][1], x.x, x.y, k.x, k.y);
          mma16816_top(s[t][0], s[t][1], x.z, x.w, k.z, k.w);
        }
      }
      load_k(j0 + kWarps * 16);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[t][e] = j0 + t * 8 + 2 * c + e <= pos ? s[t][e] * sc : -INFINITY;
          mn = fmaxf(mn, s[t][e]);
        }
      }
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));  // finite: key j0 is visible
      const float corr = exp2f(m - mn);
      m = mn;
      l *= corr;
#pragma unroll
      for (int p = 0; p < PANELS; ++p)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[p][j][0] *= corr;
          acc[p][j][1] *= corr;
        }
      uint32_t hi[2], lo[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float x = exp2f(s[t][0] - mn), y = exp2f(s[t][1] - mn);
        l += x + y;
        hi[t] = pack2(x, y);
        const float2 f = unpack2(hi[t]);
        lo[t] = pack2(x - f.x, y - f.y);
      }
#pragma unroll
      for (int p = 0; p < PANELS; ++p) {
        const uint32_t v[4][4] = {{vr[0][p].x, vr[0][p].y, vr[0][p].z, vr[0][p].w}, {vr[1][p].x, vr[1][p].y, vr[1][p].z, vr[1][p].w},
                                  {vr[2][p].x, vr[2][p].y, vr[2][p].z, vr[2][p].w}, {vr[3][p].x, vr[3][p].y, vr[3][p].z, vr[3][p].w}};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;  // element j of two keys
          const uint32_t b0 = __byte_perm(v[0][j >> 1], v[1][j >> 1], sel), b1 = __byte_perm(v[2][j >> 1], v[3][j >> 1], sel);
          mma16816_top(acc[p][j][0], acc[p][j][1], hi[0], hi[1], b0, b1);
          mma16816_top(acc[p][j][0], acc[p][j][1], lo[0], lo[1], b0, b1);
        }
      }
      load_v(j0 + kWarps * 16);
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const int pitch = PANELS * 64 + 2;  // per warp and head: P*V, maximum, sum
    float* mine = sm + (warp * 8 + g) * pitch;
    __syncthreads();                    // the previous item's merge has been read
    if (g < G) {
#pragma unroll
      for (int p = 0; p < PANELS; ++p)
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // columns 2c, 2c + 1 of MMA j
          mine[p * 64 + 16 * c + j] = acc[p][j][0];
          mine[p * 64 + 16 * c + 8 + j] = acc[p][j][1];
        }
      if (c == 0) {
        mine[PANELS * 64] = m;
        mine[PANELS * 64 + 1] = l;
      }
    }
    __syncthreads();
    const int used = min(kWarps, pos / 16 + 1);  // warps that had keys
#pragma unroll 1
    for (int i = threadIdx.x; i < G * a.hd / 2; i += kThreads) {
      const int h = (2 * i) / a.hd, d = 2 * i - h * a.hd;
      const float* from = sm + h * pitch;
      float mx = -INFINITY;
#pragma unroll 4
      for (int w = 0; w < used; ++w) mx = fmaxf(mx, from[w * 8 * pitch + PANELS * 64]);
      float ls = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 4
      for (int w = 0; w < used; ++w) {
        const float* x = from + w * 8 * pitch;
        const float f = exp2f(x[PANELS * 64] - mx);
        ls += x[PANELS * 64 + 1] * f;
        o0 += x[d] * f;
        o1 += x[d + 1] * f;
      }
      const uint32_t v = pack2(o0 / ls, o1 / ls);
      const size_t at = (size_t)b * (qd / 2) + (size_t)((h0 + h) * a.hd + d) / 2;
      if constexpr (R8 == 1) put_word(a.w_att + at, v, epoch);
      else __stcg(reinterpret_cast<unsigned*>(a.att) + at, v);
    }
  }
}

__device__ __forceinline__ unsigned long long pack_best(float v, int i) {  // larger value first, then the lower index
  uint32_t u = __float_as_uint(v);
  u ^= (u >> 31) ? 0xffffffffu : 0x80000000u;
  return ((unsigned long long)u << 32) | (0xffffffffu - (uint32_t)i);
}
__device__ __forceinline__ float best_value(unsigned long long k) {
  const uint32_t u = (uint32_t)(k >> 32);
  return __uint_as_float((u >> 31) ? u ^ 0x80000000u : ~u);
}

template <int R8>
__global__ void __launch_bounds__(kThreads, 1) decode_steps_kernel(const __grid_constant__ DecodeArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_tok[32], s_abort;
  __shared__ float s_sq[2 * kWarps], s_cos[64], s_sin[64];
  __shared__ __align__(8) uint64_t s_full[Ring<R8>::kSlots];
  __shared__ unsigned long long s_best[32];
  __shared__ double s_before[32], s_target[32];
  __shared__ Prod s_prod[5];
  constexpr int BP = 8 * R8, J = kThreads / BP;  // a thread's row of the batch is fixed: threadIdx.x % BP
  constexpr bool kWords = R8 == 1;
  uint8_t* stage = smem;
  float2* part = reinterpret_cast<float2*>(smem + a.stage_bytes + Ring<R8>::kSlots * a.slot_bytes);  // staged rows | ring of weights | partial sums
  const int row = threadIdx.x & (BP - 1), j0 = threadIdx.x / BP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = a.D, QD = a.H * a.hd, KVD = a.KV * a.hd;
  const bool sampling = a.temperature > 1e-6f, live = row < a.B;
  if (threadIdx.x == 0) {
    s_abort = 0;
    make_prod(s_prod[kQkv], kQkv, a.off_qkv, a.layer_stride, D, (QD + 2 * KVD) / 8);
    make_prod(s_prod[kWo], kWo, a.off_wo, a.layer_stride, QD, D / 8);
    make_prod(s_prod[kW13], kW13, a.off_w13, a.layer_stride, D, 2 * a.Hd / 8);
    make_prod(s_prod[kW2], kW2, a.off_w2, a.layer_stride, a.Hd, D / 8);
    make_prod(s_prod[kHead], kHead, a.off_embed, 0, D, a.V / 8);
  }
  for (int i = threadIdx.x * 16; i < a.stage_bytes; i += kThreads * 16) *reinterpret_cast<uint4*>(stage + i) = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const Wait wait{a.status, &s_abort};
  GridBarrier bar{a.bar, 0u, wait};
  RowShare share;
  share.per_row = a.B >= 16 ? 1 : kWarps / a.B;
  share.row = warp / share.per_row;
  share.sub = warp - share.row * share.per_row;
  constexpr int kFeeder = kThreads - 32;
  Feed<R8> feed{smem_u32(s_full), smem_u32(smem) + (uint32_t)a.stage_bytes, a.slot_bytes, 0, 0, 1, 0, 0};
  if (threadIdx.x == kFeeder) {
    for (int i = 0; i < Ring<R8>::kSlots; ++i) mbar_init(feed.bar + 8u * i, 1);
    fence_mbar_init();
    feed.issue(a, s_prod);
  }
  __syncthreads();
  int group = 0;  // groups consumed
  auto group_ready = [&] {
    if (!mbar_wait(feed.bar + 8u * (group % Ring<R8>::kSlots), (uint32_t)(group / Ring<R8>::kSlots) & 1u, a.status, DEV_GRID_TIMEOUT)) s_abort = 1;
  };
  // every way out before the end: no copy may still be on its way into this CTA's shared memory
  auto leave = [&] {
    if (threadIdx.x == kFeeder)
      for (int i = feed.used; i < feed.issued; ++i)
        mbar_wait(feed.bar + 8u * (i % Ring<R8>::kSlots), (uint32_t)(i / Ring<R8>::kSlots) & 1u, nullptr, 0);
  };

#pragma unroll 1
  for (int step = 1; step < a.n_new; ++step) {
    const int pos = a.prompt + step - 1;
    unsigned long long* best = a.best + (step % 3) * a.B;
    if ((int)threadIdx.x < a.B) {
      int t;
      if (step == 1 || sampling) {
        t = (int)__ldcg(a.tok + threadIdx.x);
      } else {
        const unsigned long long k = __ldcg(a.best + ((step - 1) % 3) * a.B + threadIdx.x);
        t = k == 0 ? 0 : (int)(0xffffffffu - (uint32_t)k);
        if (blockIdx.x == 0) a.out[(size_t)threadIdx.x * a.n_new + step - 1] = (uint16_t)t;
      }
      s_tok[threadIdx.x] = t;
      // the next step's slot: last read at the start of the step before, written after this step's barrier
      if (blockIdx.x == 0) __stcg(a.best + ((step + 1) % 3) * a.B + threadIdx.x, 0ull);
    }
    if (threadIdx.x < 32) s_best[threadIdx.x] = 0;
    if ((int)threadIdx.x < a.hd / 2) {
      s_cos[threadIdx.x] = a.cosb[pos * (a.hd / 2) + threadIdx.x];
      s_sin[threadIdx.x] = a.sinb[pos * (a.hd / 2) + threadIdx.x];
    }
    __syncthreads();
    float bv = -INFINITY;
    int bi = -1;
    // the products of the step in order: q|k|v (then attention), Wo, W1|W3, W2 of every layer, and the classifier
#pragma unroll 1
    for (int idx = 0; idx <= 4 * a.L; ++idx) {
      const int l = idx >> 2, kind = l == a.L ? kHead : idx & 3;
      const Prod& p = s_prod[kind];
      const uint32_t epoch = (uint32_t)(step * a.L + l + 1);
      const bool direct = kind == kWo || kind == kW2;
      if (R8 > 1 && kind == kQkv) {
        // The cached keys and values that this CTA will attend to, from DRAM into L2 while q|k|v are computed: 164 KB per
        // item at 640 positions, more than all of it fits at once, and the attention's own loads are a chain of a few.
        const int group_heads = a.group, hgroups = a.H / group_heads, row_bytes = a.hd * 2, lines = (row_bytes + 127) / 128;
        for (int item = blockIdx.x; item < a.B * hgroups; item += gridDim.x) {
          const int b = item / hgroups, kvh = (item - b * hgroups) * group_heads / (a.H / a.KV);
          const size_t base = (size_t)l * a.kv_layer + (size_t)b * a.S * KVD + (size_t)kvh * a.hd;
          for (int i = threadIdx.x; i < 2 * pos * lines; i += kThreads) {
            const int j = i / (2 * lines), part = i - j * 2 * lines;
            const bf16* from = (part < lines ? a.kcache : a.vcache) + base + (size_t)j * KVD + (part % lines) * 64;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(from));
          }
        }
      }
      Source src{nullptr, nullptr, nullptr, a.B, epoch};
      float2 old = make_float2(0.f, 0.f);  // residual of this thread's first pair
      const float* xrow = kind == kWo && l == 0 ? a.p + a.off_embed_f32 + (size_t)s_tok[live ? row : 0] * D : a.x + (size_t)row * D;
      const uint2* wrow = (kind == kWo ? a.w_x0 : a.w_x1) + (size_t)row * D;
      auto residual = [&](int col) {
        if (!kWords || (kind == kWo && l == 0)) return __ldcg(reinterpret_cast<const float2*>(xrow + col));
        const uint4 o = get_words(wrow + col);  // complete: this CTA has staged it
        return make_float2(__uint_as_float(o.x), __uint_as_float(o.z));
      };
      if (direct) {
        if (kWords) __syncthreads();  // the partial sums of the phase before have been read
        src.rows = kind == kWo ? a.att : a.gate;
        src.words = kind == kWo ? a.w_att : a.w_gate;
        if (live && j0 < p.nu * 4) old = residual(p.row0(j0 >> 2) + 2 * (j0 & 3));
      } else {
        // x before this layer (after W2 of the one below; the embedding row for layer 0), or after Wo for W1|W3
        const bool embed = kind == kQkv && l == 0;
        const uint2* words = !kWords || embed ? nullptr : kind == kW13 ? a.w_x1 : a.w_x0;
        group_ready();
        const float* gains = reinterpret_cast<const float*>(smem + a.stage_bytes + (group % Ring<R8>::kSlots + 1) * a.slot_bytes - D * 4);
        stage_norm<R8>(D, a.B, [&](int r) { return embed ? a.p + a.off_embed_f32 + (size_t)s_tok[r] * D : a.x + (size_t)r * D; }, words,
                       kind == kW13 ? epoch : epoch - 1, gains, stage, s_sq, share, wait);
        __syncthreads();
        src.stage = reinterpret_cast<const uint4*>(stage);
      }
      {
        const Share mine = make_share(p.K);
        uint4 frag[4][R8];
#pragma unroll 1
        for (int g0 = 0; g0 < p.nu; g0 += Ring<R8>::kUnits, ++group) {
          const int n = min(Ring<R8>::kUnits, p.nu - g0);
          group_ready();
          run_units<R8>(mine, n, smem + a.stage_bytes + (group % Ring<R8>::kSlots) * a.slot_bytes, part, src, frag, g0 == 0, wait);
          __syncthreads();
          if (threadIdx.x == kFeeder) {  // the slot is free: refill it
            ++feed.used;
            feed.issue(a, s_prod);
          }
          if (live) {
            if (kind == kW13) {
#pragma unroll 1
              for (int i = j0; i < n * 2; i += J) {
                const int u = (i >> 2) * 2, c = i & 3;
                const float2 h1 = pair_sum<R8>(part, u, row, c), h3 = pair_sum<R8>(part, u + 1, row, c);
                const uint32_t g = pack2(h1.x * h3.x * sigmoid(h1.x), h1.y * h3.y * sigmoid(h1.y));
                const int pair = (int)blockIdx.x + ((g0 + u) >> 1) * (int)gridDim.x;  // columns 8 pair .. of the gate
                const size_t at = (size_t)row * (a.Hd / 2) + pair * 4 + c;
                if (kWords) put_word(a.w_gate + at, g, epoch);
                else __stcg(reinterpret_cast<unsigned*>(a.gate) + at, g);
              }
            } else {
#pragma unroll 1
              for (int i = j0; i < n * 4; i += J) {
                const float2 s = pair_sum<R8>(part, i >> 2, row, i & 3);
                const int col = p.row0(g0 + (i >> 2)) + 2 * (i & 3);
                float x = s.x, y = s.y;
                if (kind == kQkv) {
                  if (col < QD + KVD) {
                    const int r = (col - (int)__umulhi((unsigned)col, a.hd_magic) * a.hd) >> 1;
                    const float c = s_cos[r], sn = s_sin[r];
                    const float t = x * c - y * sn;
                    y = y * c + x * sn;
                    x = t;
                  }
                  const uint32_t v = pack2(x, y);
                  if (kWords) put_word(a.w_qkv + (size_t)row * ((QD + 2 * KVD) / 2) + col / 2, v, epoch);
                  else if (col < QD) __stcg(reinterpret_cast<unsigned*>(a.q + (size_t)row * QD + col), v);
                  if (col >= QD) {
                    bf16* cache = (col < QD + KVD ? a.kcache + (col - QD) : a.vcache + (col - QD - KVD)) + (size_t)l * a.kv_layer;
                    __stcg(reinterpret_cast<unsigned*>(cache + ((size_t)row * a.S + pos) * KVD), v);
                  }
                } else if (kind == kHead) {
                  if (x > bv) { bv = x; bi = col; }
                  if (y > bv) { bv = y; bi = col + 1; }
                  if (sampling) __stcg(reinterpret_cast<float2*>(a.logits + (size_t)row * a.V + col), s);
                } else {  // x += product; every element is updated by one thread
                  const size_t at = (size_t)row * D + col;
                  if (g0 > 0 || i != j0) old = residual(col);
                  x += old.x;
                  y += old.y;
                  if (kWords) {
                    uint2* to = (kind == kWo ? a.w_x1 : a.w_x0) + at;
                    put_word(to, __float_as_uint(x), epoch);
                    put_word(to + 1, __float_as_uint(y), epoch);
                  } else {
                    __stcg(reinterpret_cast<float2*>(a.x + at), make_float2(x, y));
                  }
                }
              }
            }
          }
          if (g0 + n < p.nu) __syncthreads();
        }
      }
      if (kWords ? s_abort != 0 : kind != kHead && !bar.sync()) {
        leave();
        return;
      }
      if (kind == kQkv) {
        const size_t cl = (size_t)l * a.kv_layer;
        float* sm = reinterpret_cast<float*>(part);
        if (a.hd <= 64) attention_phase<R8, 1>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
        else attention_phase<R8, 2>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
        if (!kWords && !bar.sync()) {
          leave();
          return;
        }
      }
    }
    // ---- the best logit of every row
    if (bi >= 0) atomicMax(&s_best[row], pack_best(bv, bi));
    __syncthreads();
    if ((int)threadIdx.x < a.B && s_best[threadIdx.x] != 0) atomicMax(best + threadIdx.x, s_best[threadIdx.x]);
    if (!bar.sync()) {
      leave();
      return;
    }
    if (!sampling) continue;
    // ---- temperature sampling (ane/train_full.go:318-342): this CTA's vocabulary range of every row in double, the
    // ranges' sums in order, and the CTA whose range holds the target walks it
    const Prod& head = s_prod[kHead];
    const int v0 = head.u0 * 8, v1 = (head.u0 + head.nu) * 8;
    const double inv_temp = (double)(1.0f / a.temperature);
#pragma unroll 1
    for (int b = warp; b < a.B; b += kWarps) {
      const double mx = (double)best_value(__ldcg(best + b));
      double s = 0.0;
#pragma unroll 1
      for (int v = v0 + lane; v < v1; v += 32) s += exp(((double)__ldcg(a.logits + (size_t)b * a.V + v) - mx) * inv_temp);
      s = warp_sum_d(s);
      if (lane == 0) __stcg(a.psum + (size_t)blockIdx.x * a.B + b, s);
    }
    if (!bar.sync()) {
      leave();
      return;
    }
    double* s_sums = reinterpret_cast<double*>(part);  // [gridDim.x][B]
#pragma unroll 1
    for (int i = threadIdx.x; i < (int)gridDim.x * a.B; i += kThreads) s_sums[i] = __ldcg(a.psum + i);
    __syncthreads();
    if ((int)threadIdx.x < a.B) {
      double total = 0.0;
#pragma unroll 4
      for (int c = 0; c < (int)gridDim.x; ++c) total += s_sums[c * a.B + threadIdx.x];
      const double target = a.u[(size_t)step * a.u_stride + threadIdx.x] * total;
      double acc = 0.0, before = 0.0;
      int owner = -1;
#pragma unroll 1
      for (int c = 0; c < (int)gridDim.x; ++c) {
        before = acc;
        acc += s_sums[c * a.B + threadIdx.x];
        const long long units = a.V / 8;  // a CTA without vocabulary cannot own the target
        if (acc >= target && c * units / (int)gridDim.x < (c + 1) * units / (int)gridDim.x) {
          owner = c;
          break;
        }
      }
      s_tok[threadIdx.x] = owner == (int)blockIdx.x;
      s_before[threadIdx.x] = before;
      s_target[threadIdx.x] = target;
      if (owner < 0 && blockIdx.x == 0) {  // the running sum never reaches the target: the last index
        a.tok[threadIdx.x] = (uint16_t)(a.V - 1);
        a.out[(size_t)threadIdx.x * a.n_new + step] = (uint16_t)(a.V - 1);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int b = warp; b < a.B; b += kWarps) {
      if (!s_tok[b]) continue;
      const double mx = (double)best_value(__ldcg(best + b));
      double acc = s_before[b];
      int pick = v1 - 1;
#pragma unroll 1
      for (int v = v0; v < v1; v += 32) {
        double e = v + lane < v1 ? exp(((double)__ldcg(a.logits + (size_t)b * a.V + v + lane) - mx) * inv_temp) : 0.0;
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {  // inclusive scan
          const double t = __shfl_up_sync(0xffffffffu, e, o);
          if (lane >= o) e += t;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, acc + e >= s_target[b] && v + lane < v1);
        if (hit) {
          pick = v + __ffs(hit) - 1;
          break;
        }
        acc += __shfl_sync(0xffffffffu, e, 31);
      }
      if (lane == 0) {
        a.tok[b] = (uint16_t)pick;
        a.out[(size_t)b * a.n_new + step] = (uint16_t)pick;
      }
    }
    if (!bar.sync()) {
      leave();
      return;
    }
  }
  if (!sampling && a.n_new > 1 && blockIdx.x == 0 && (int)threadIdx.x < a.B) {
    const unsigned long long k = __ldcg(a.best + ((a.n_new - 1) % 3) * a.B + threadIdx.x);
    a.out[(size_t)threadIdx.x * a.n_new + a.n_new - 1] = (uint16_t)(k == 0 ? 0 : 0xffffffffu - (uint32_t)k);
  }
}

size_t stage_bytes(int r8, int D) { return (size_t)((D + 31) / 32) * r8 * 512; }
// a group's units with the norm's gains behind them, or the W2 units of a CTA (mostly one)
size_t slot_bytes(int r8, int D, int Hd, int ctas) {
  const int units = r8 == 4 ? Ring<4>::kUnits : Ring<2>::kUnits, w2 = std::min(units, (D / 8 + ctas - 1) / ctas);
  return std::max((size_t)16 * w2 * Hd, (size_t)16 * units * D + 4 * D);
}
size_t tail_bytes(int r8, int hd, int ctas, int B) {  // partial sums; the attention merge and the sampler's sums use the same memory
  const size_t unit = sizeof(float2) * kWarps * (size_t)(r8 == 1 ? Part<1>::kVecs : r8 == 2 ? Part<2>::kVecs : Part<4>::kVecs);
  return std::max(unit * (r8 == 4 ? Ring<4>::kUnits : Ring<2>::kUnits),
                  std::max(sizeof(float) * (size_t)(kWarps * 8 * (2 + (hd <= 64 ? 64 : 128))), sizeof(double) * (size_t)ctas * B));
}
size_t smem_bytes(int r8, int D, int Hd, int hd, int ctas, int B) {
  return stage_bytes(r8, D) + (r8 == 4 ? Ring<4>::kSlots : Ring<2>::kSlots) * slot_bytes(r8, D, Hd, ctas) + tail_bytes(r8, hd, ctas, B);
}
constexpr size_t kSmemLimit = 224 * 1024;  // beside the static arrays

int row_groups(int batch) { return batch <= 8 ? 1 : batch <= 16 ? 2 : 4; }

}  // namespace

// The exchange of flagged words needs every CTA to own units of q|k|v and of W1|W3; more CTAs than that would idle anyway.
// A multiple of 4: see Prod.
static int decode_ctas(int sms, int Hd, int H, int KV, int hd) { return std::min(std::min(sms, 148), std::min((H + 2 * KV) * hd / 8, Hd / 8)) & ~3; }

bool decode_steps_supported(int D, int Hd, int H, int KV, int hd, int V, int batch, int sms) {
  const int ctas = decode_ctas(sms, Hd, H, KV, hd);
  return batch >= 1 && batch <= 32 && hd % 8 == 0 && hd <= 128 && D % 8 == 0 && H * hd == D && Hd % 32 == 0 && V % 8 == 0 && H % KV == 0 &&
         ctas > 0 && smem_bytes(row_groups(batch), D, Hd, hd, ctas, batch) <= kSmemLimit;
}
size_t decode_words_bytes(int D, int Hd, int H, int KV, int hd) {  // exchange buffers of up to 8 sequences
  return sizeof(uint2) * 8 * ((size_t)2 * D + (size_t)(H + 2 * KV) * hd / 2 + (size_t)H * hd / 2 + (size_t)Hd / 2);
}

int decode_steps(DecodeArgs a, void* words, int sms, cudaStream_t s) {
  if (a.n_new < 2) return 0;
  const int r8 = row_groups(a.B), qd = a.H * a.hd, qkv = (a.H + 2 * a.KV) * a.hd;
  a.stage_bytes = (int)stage_bytes(r8, a.D);
  const int ctas = decode_ctas(sms, a.Hd, a.H, a.KV, a.hd);
  a.slot_bytes = (int)slot_bytes(r8, a.D, a.Hd, ctas);
  const int rep = a.H / a.KV;
  a.group = rep <= 8 ? rep : 1;  // query heads per attention item: rows of one fragment
  a.hd_magic = 0xffffffffu / (unsigned)a.hd + 1u;  // col / hd = umulhi(col, hd_magic) for col < 2^16
  uint2* p = reinterpret_cast<uint2*>(words);
  a.w_x0 = p; p += (size_t)8 * a.D;
  a.w_x1 = p; p += (size_t)8 * a.D;
  a.w_qkv = p; p += (size_t)8 * qkv / 2;
  a.w_att = p; p += (size_t)8 * qd / 2;
  a.w_gate = p;
  const size_t bytes = smem_bytes(r8, a.D, a.Hd, a.hd, ctas, a.B);
  auto kern = r8 == 1 ? decode_steps_kernel<1> : r8 == 2 ? decode_steps_kernel<2> : decode_steps_kernel<4>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return -3;
  if (cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s) != cudaSuccess ||
      cudaMemsetAsync(words, 0, decode_words_bytes(a.D, a.Hd, a.H, a.KV, a.hd), s) != cudaSuccess ||
      cudaMemsetAsync(a.best, 0, 3 * sizeof(unsigned long long) * (size_t)a.B, s) != cudaSuccess)
    return -3;
  void* args[] = {&a};
  // cooperative: all CTAs are resident together, so the waits on one another complete
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(ctas), dim3(kThreads), args, bytes, s) == cudaSuccess ? 0 : -4;
}

}  // namespace ane
