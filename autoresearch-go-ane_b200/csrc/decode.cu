// KV-cached generation: all steps after the prefill in ONE persistent cooperative kernel (llama-style architecture,
// bf16 engines).
//
// A decode step is about sixty dependent products with at most 32 rows.  Launched one by one each of them costs the
// fixed latency of a kernel (a 128-row tensor-core tile of the training GEMM takes 10-15 us for 8 KB of useful output),
// although the bytes of a step -- every weight once, keys and values once -- take 35-75 us at the memory's rate.  Here
// one CTA per SM stays resident and walks through the five phases of a layer (q|k|v, attention, Wo, W1|W3, W2).  What
// bounds it is the latency of a phase: how fast one SM's results reach all others, and the chain of instructions
// between reading activations and publishing results.  So:
//   * Weights never change: each warp requests its share of the NEXT phase's weights (cp.async) before it waits
//     for that phase's activations, so the weight stream runs under the exchange.
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
// lane requests 16 contiguous bytes of a weight row (k = 8 (lane % 4) ..) and uses them as the fragments of two MMAs: no
// ldmatrix, and nobody else ever reads its slot.
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

// 16 bytes of a weight row into this lane's slot of the ring (zeros instead when `in` is false); past L1
__device__ __forceinline__ void request_weight(uint32_t slot, const bf16* p, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot), "l"(p), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void requests_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void requests_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Values that other SMs wrote earlier in this kernel: L2 only.
__device__ __forceinline__ uint4 ld_l2(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

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
// One product's share of this CTA (in shared memory): `nu` units of 8 weight rows.
struct Prod {
  size_t off, layer_stride;
  int K, nu, u0, kind;
  __device__ __forceinline__ int row0(int i) const {
    if (kind == kHead) return (u0 + i) * 8;  // a contiguous range of the vocabulary
    if (kind != kW13) return ((int)blockIdx.x + i * (int)gridDim.x) * 8;
    // W1 and W3 lie in blocks of 32 rows; units 2j and 2j+1 are matching rows of the two
    const int p = (int)blockIdx.x + (i >> 1) * (int)gridDim.x;
    return (p >> 2) * 64 + (p & 3) * 8 + (i & 1) * 32;
  }
};
__device__ __forceinline__ void make_prod(Prod& d, int kind, size_t off, size_t layer_stride, int K, int n_units) {
  const int g = (int)gridDim.x, b = (int)blockIdx.x;
  d.off = off;
  d.layer_stride = layer_stride;
  d.K = K;
  d.kind = kind;
  d.u0 = 0;
  if (kind == kHead) {
    d.u0 = (int)((long long)n_units * b / g);
    d.nu = (int)((long long)n_units * (b + 1) / g) - d.u0;
  } else if (kind == kW13) {
    const int pairs = n_units / 2;
    d.nu = b < pairs ? 2 * ((pairs - b + g - 1) / g) : 0;
  } else {
    d.nu = b < n_units ? (n_units - b + g - 1) / g : 0;
  }
}

// A warp's walk over the weights of units [first, first + n) of a product.  Eight 16-byte vectors per lane are in
// flight, each in a shared-memory slot of its lane (registers would be spilled while activations are staged, and a
// spill waits for its load): four units of up to two 32-wide chunks, or two units of up to four chunks (longer
// contractions block by block).
constexpr int kSlots = 8;
constexpr int kRingBytes = kWarps * kSlots * 512;
struct Walk {
  uint32_t ring;       // this lane's first slot
  const bf16* base;    // weights + this lane's column
  int K, k0, nc;       // this lane's first column, this warp's chunks
  int unit, end, blk;  // next to request
  template <int NCB>
  __device__ __forceinline__ void request(const Prod& p, int slot) {
    if (unit < end) {  // warp-uniform
      const int lane = threadIdx.x & 31;
      const bf16* q = base + (size_t)(p.row0(unit) + (lane >> 2)) * K + blk * 128;
      const int k = k0 + blk * 128, left = nc - blk * 4;
#pragma unroll
      for (int c = 0; c < NCB; ++c) {
        const bool in = k + c * 32 < K;
        if (c < left) request_weight(ring + (uint32_t)(slot + c) * 512u, in ? q + c * 32 : q, in);
      }
      if (NCB == 2 || ++blk * 4 >= nc) {
        blk = 0;
        ++unit;
      }
    }
    requests_commit();  // one group per block, empty or not
  }
  __device__ __forceinline__ void start(const Prod& p, const bf16* w, int first, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    K = p.K;
    const int chunks = (K + 31) >> 5, per = (chunks + kWarps - 1) / kWarps, c0 = min(warp * per, chunks);
    nc = min(per, chunks - c0);
    k0 = c0 * 32 + (lane & 3) * 8;
    base = w + k0;
    unit = first;
    end = nc > 0 ? first + n : 0;
    blk = 0;
    if (nc <= 2) {
#pragma unroll 1
      for (int i = 0; i < kSlots; i += 2) request<2>(p, i);
    } else {
#pragma unroll 1
      for (int i = 0; i < kSlots; i += 4) request<4>(p, i);
    }
  }
};

// Where a warp's A fragments come from: normalised rows staged in shared memory (read once per product when two chunks
// or fewer), or, for Wo and W2 (no norm, and mostly one unit per CTA), straight from the exchanged bf16 rows.
template <int R8>
struct StagedRows {
  const uint4* stage;
  template <int NCB>
  __device__ __forceinline__ void read(uint4 (&f)[NCB][R8], const Walk& w, int first) const {
    const uint4* st = stage + (size_t)((w.k0 >> 5) + first) * R8 * 32 + (threadIdx.x & 31);
#pragma unroll
    for (int c = 0; c < NCB; ++c)
#pragma unroll
      for (int r = 0; r < R8; ++r)
        if (c < w.nc - first) f[c][r] = st[(c * R8 + r) * 32];
  }
};
template <int R8>
struct PlainRows {
  const bf16* rows;
  int B;
  template <int NCB>
  __device__ __forceinline__ void read(uint4 (&f)[NCB][R8], const Walk& w, int first) const {
    const int g = (threadIdx.x & 31) >> 2;
#pragma unroll
    for (int c = 0; c < NCB; ++c) {
      const int k = w.k0 + (first + c) * 32;
      const bool in = c < w.nc - first && k < w.K;
#pragma unroll
      for (int r = 0; r < R8; ++r) {
        const bool ok = in && r * 8 + g < B;
        f[c][r] = ok ? ld_l2(rows + (size_t)(r * 8 + g) * w.K + k) : make_uint4(0, 0, 0, 0);
      }
    }
  }
};
struct WordRows {  // R8 = 1; words {two values, epoch}
  const uint2* words;
  int B;
  uint32_t epoch;
  Wait wait;
  template <int NCB>
  __device__ __forceinline__ void read(uint4 (&f)[NCB][1], const Walk& w, int first) const {
    const int g = (threadIdx.x & 31) >> 2;
    long long t0 = 0;
#pragma unroll 1
    for (unsigned n = 0;; ++n) {
      bool ok = true;
#pragma unroll
      for (int c = 0; c < NCB; ++c) {
        const int k = w.k0 + (first + c) * 32;
        uint4 x = make_uint4(0, epoch, 0, epoch), y = x;
        if (c < w.nc - first && k < w.K && g < B) {
          const uint2* p = words + ((size_t)g * w.K + k) / 2;
          x = get_words(p);
          y = get_words(p + 2);
        }
        ok = ok && x.y == epoch && x.w == epoch && y.y == epoch && y.w == epoch;
        f[c][0] = make_uint4(x.x, x.z, y.x, y.z);
      }
      if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) return;
    }
  }
};

// Partial sums of the n units the walk was started on: this warp's chunks.
template <int R8, int NCB, class Rows>
__device__ __forceinline__ void run_units(const Prod& p, Walk& w, int n, float2* part, const Rows& rows) {
  constexpr int T = (R8 + 1) / 2, BLOCKS = kSlots / NCB;
  using P = Part<R8>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* d = part + (size_t)warp * P::kVecs + (lane & 3) * P::kPitch + (lane >> 2);
  float acc[T][4] = {};
  constexpr int NA = NCB == 4 && R8 == 4 ? 2 : NCB;  // chunks whose A fragments are held together (registers)
  uint4 a[NA][R8];
  if (NCB == 2) rows.template read<NA>(a, w, 0);  // all chunks of this warp: the same for every unit
  int unit = 0, blk = 0, slot = 0;
#pragma unroll 1
  while (unit < n) {
    if (NCB == 4) rows.template read<NA>(a, w, blk * 4);
    requests_wait<BLOCKS - 1>();
    const int left = w.nc - blk * 4;
#pragma unroll
    for (int c = 0; c < NCB; ++c) {
      if (NA < NCB && c == NA) rows.template read<NA>(a, w, blk * 4 + NA);
      if (c < left) {
        uint4 b;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(w.ring + (uint32_t)(slot + c) * 512u) : "memory");
#pragma unroll
        for (int t = 0; t < T; ++t) {
          const uint4 lo = a[c % NA][2 * t], hi = R8 > 1 ? a[c % NA][R8 > 1 ? 2 * t + 1 : 0] : make_uint4(0, 0, 0, 0);
          mma16816(acc[t], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
          mma16816(acc[t], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
        }
      }
    }
    w.request<NCB>(p, slot);
    slot = (slot + NCB) & (kSlots - 1);
    if (NCB == 2 || ++blk * 4 >= w.nc) {
      blk = 0;
#pragma unroll
      for (int t = 0; t < T; ++t) {
        d[t * P::kTile] = make_float2(acc[t][0], acc[t][1]);
        if (R8 > 1) d[t * P::kTile + 8] = make_float2(acc[t][2], acc[t][3]);
        acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
      }
      d += kWarps * P::kVecs;
      ++unit;
    }
  }
}
template <int R8, class Rows>
__device__ __forceinline__ void run_product(const Prod& p, Walk& w, int n, float2* part, const Rows& rows) {
  if (w.nc <= 2) run_units<R8, 2>(p, w, n, part, rows);
  else run_units<R8, 4>(p, w, n, part, rows);
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

// A warp holds one row in segments of 768 columns, 24 values per lane: plain fp32 as six float4, words as twelve pairs.
constexpr int kSeg = 768;
struct RowSeg {
  float v[24];
};
// plain: values 4 i .. 4 i + 3 are columns k0 + 4 (lane + 32 i)
__device__ __forceinline__ void read_plain(RowSeg& x, const float* row, int k0, int K) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const int k = k0 + 4 * (lane + 32 * i);
    const float4 f = k < K ? __ldcg(reinterpret_cast<const float4*>(row + k0 + 4 * lane) + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    x.v[4 * i] = f.x; x.v[4 * i + 1] = f.y; x.v[4 * i + 2] = f.z; x.v[4 * i + 3] = f.w;
  }
}
// words: values 2 i, 2 i + 1 are columns k0 + 2 (lane + 32 i)
__device__ __forceinline__ void read_words(RowSeg& x, const uint2* row, int k0, int K, uint32_t epoch, const Wait& wait) {
  const int lane = threadIdx.x & 31;
  long long t0 = 0;
#pragma unroll 1
  for (unsigned n = 0;; ++n) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const int k = k0 + 2 * (lane + 32 * i);
      uint4 u = make_uint4(0, epoch, 0, epoch);
      if (k < K) u = get_words(row + k0 + 2 * lane + 64 * i);
      ok = ok && u.y == epoch && u.w == epoch;
      x.v[2 * i] = __uint_as_float(u.x);
      x.v[2 * i + 1] = __uint_as_float(u.z);
    }
    if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) return;
  }
}
// the norm's weights of the same columns
template <bool WORDS>
__device__ __forceinline__ void read_gains(RowSeg& g, const float* __restrict__ wn, int k0, int K) {
  const int lane = threadIdx.x & 31;
  if constexpr (WORDS) {
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float2 f = k0 + 2 * (lane + 32 * i) < K ? __ldg(reinterpret_cast<const float2*>(wn + k0 + 2 * lane) + 32 * i) : make_float2(0.f, 0.f);
      g.v[2 * i] = f.x; g.v[2 * i + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float4 f = k0 + 4 * (lane + 32 * i) < K ? __ldg(reinterpret_cast<const float4*>(wn + k0 + 4 * lane) + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
      g.v[4 * i] = f.x; g.v[4 * i + 1] = f.y; g.v[4 * i + 2] = f.z; g.v[4 * i + 3] = f.w;
    }
  }
}
template <int R8, bool WORDS>
__device__ __forceinline__ void put_seg(const RowSeg& x, float rms, const RowSeg& g, int r, int k0, int K, uint8_t* stage) {
  const int lane = threadIdx.x & 31;
  if constexpr (WORDS) {
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const int k = k0 + 2 * (lane + 32 * i);
      if (k < K) *reinterpret_cast<uint32_t*>(stage + frag_at<R8>(r, k)) = pack2(x.v[2 * i] * rms * g.v[2 * i], x.v[2 * i + 1] * rms * g.v[2 * i + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int k = k0 + 4 * (lane + 32 * i);
      if (k < K)
        *reinterpret_cast<uint2*>(stage + frag_at<R8>(r, k)) =
            make_uint2(pack2(x.v[4 * i] * rms * g.v[4 * i], x.v[4 * i + 1] * rms * g.v[4 * i + 1]),
                       pack2(x.v[4 * i + 2] * rms * g.v[4 * i + 2], x.v[4 * i + 3] * rms * g.v[4 * i + 3]));
    }
  }
}
// Normalised rows, bf16(x * rms^-1 * w), rounded like the training forward's: warp w takes rows w and w + 16.
template <int R8, bool WORDS, class Row>
__device__ __forceinline__ void stage_norm(int K, int B, Row row, uint32_t epoch, const float* __restrict__ wn, uint8_t* stage, const Wait& wait) {
  const int warp = threadIdx.x >> 5;
  RowSeg x, gain;
  auto read = [&](int r, int k0) {
    if constexpr (WORDS) read_words(x, row(r), k0, K, epoch, wait);
    else read_plain(x, row(r), k0, K);
  };
  auto squares = [&] {
    float q[4] = {};
#pragma unroll
    for (int e = 0; e < 24; ++e) q[e & 3] += x.v[e] * x.v[e];
    return (q[0] + q[1]) + (q[2] + q[3]);
  };
  if (warp >= B) return;
  const bool one = K <= kSeg;
  if (one) read_gains<WORDS>(gain, wn, 0, K);  // travels together with the row
#pragma unroll 1
  for (int r = warp; r < B; r += kWarps) {
    float sq = 0.f;
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += kSeg) {
      read(r, k0);
      sq += squares();
    }
    const float rms = 1.0f / sqrtf(warp_sum(sq) / (float)K + 1e-5f);
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += kSeg) {
      if (!one) {  // wider rows are read again
        read_gains<WORDS>(gain, wn, k0, K);
        read(r, k0);
      }
      put_seg<R8, WORDS>(x, rms, gain, r, k0, K, stage);
    }
  }
}

// ---- attention ------------------------------------------------------------------------------------------------------
// One new token per sequence over cache positions 0..pos.  A work item is one sequence and G query heads of one KV head;
// its keys are dealt to groups of `lpk` lanes (8 dimensions of the head each), every group keeps its own running
// maximum, sum and P*V, and they are merged at the end.  Scores in the log2 domain.  With flagged words (R8 = 1) q and
// the new key and value come from the words, the older ones from the cache.
template <int R8, int G>
__device__ __forceinline__ void attention_phase(const DecodeArgs& a, const bf16* kc, const bf16* vc, int pos, float* sm, uint32_t epoch, const Wait& wait) {
  constexpr int U = R8 == 1 ? 2 : 4;  // keys per group in flight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lpk = a.hd <= 8 ? 1 : a.hd <= 16 ? 2 : a.hd <= 32 ? 4 : a.hd <= 64 ? 8 : 16;
  const int per_warp = 32 / lpk, groups = per_warp * kWarps;
  const int sub = lane & (lpk - 1), gid = warp * per_warp + lane / lpk;
  const bool act = sub * 8 < a.hd;
  const int d0 = act ? sub * 8 : 0;
  const int kvd = a.KV * a.hd, qd = a.H * a.hd, rep = a.H / a.KV, hgroups = a.H / G;
  const float sc = 1.4426950408889634f / sqrtf((float)a.hd);
#pragma unroll 1
  for (int item = blockIdx.x; item < a.B * hgroups; item += gridDim.x) {
    const int b = item / hgroups, h0 = (item - b * hgroups) * G, kvh = h0 / rep;
    const bf16* kb = kc + (size_t)b * a.S * kvd + (size_t)kvh * a.hd + d0;
    const bf16* vb = vc + (size_t)b * a.S * kvd + (size_t)kvh * a.hd + d0;
    uint4 kr[U], vr[U], kn = make_uint4(0, 0, 0, 0), vn = kn;
    auto fetch = [&](int j0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = min(j0 + u * groups, pos);  // clamped: a repeated key gets no weight below
        kr[u] = ld_l2(kb + (size_t)j * kvd);
        vr[u] = ld_l2(vb + (size_t)j * kvd);
      }
    };
    fetch(gid);  // cached keys do not depend on this step (R8 = 1: the newest is replaced below)
    float q[G][8];
    auto set_q = [&](int g, uint4 u) {
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack2(w[e]);
        q[g][2 * e] = act ? f.x * sc : 0.f;
        q[g][2 * e + 1] = act ? f.y * sc : 0.f;
      }
    };
    if constexpr (R8 == 1) {
      const uint2* row = a.w_qkv + (size_t)b * ((qd + 2 * kvd) / 2);
      long long t0 = 0;
  #pragma unroll 1
    for (unsigned n = 0;; ++n) {
        bool ok = true;
        auto four = [&](int col) {
          const uint4 x = get_words(row + (col >> 1)), y = get_words(row + (col >> 1) + 2);
          ok = ok && x.y == epoch && x.w == epoch && y.y == epoch && y.w == epoch;
          return make_uint4(x.x, x.z, y.x, y.z);
        };
#pragma unroll
        for (int g = 0; g < G; ++g) set_q(g, four((h0 + g) * a.hd + d0));
        kn = four(qd + kvh * a.hd + d0);
        vn = four(qd + kvd + kvh * a.hd + d0);
        if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
      }
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g) set_q(g, ld_l2(a.q + (size_t)b * qd + (size_t)(h0 + g) * a.hd + d0));
    }
    float m[G], l[G], acc[G][8];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      m[g] = -INFINITY;
      l[g] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[g][e] = 0.f;
    }
#pragma unroll 1
    for (int j0 = gid; __any_sync(0xffffffffu, j0 <= pos); j0 += groups * U) {
      if (j0 != gid) fetch(j0);
      if constexpr (R8 == 1) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (j0 + u * groups >= pos) {
            kr[u] = kn;
            vr[u] = vn;
          }
      }
      float s[U][G];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t w[4] = {kr[u].x, kr[u].y, kr[u].z, kr[u].w};
#pragma unroll
        for (int g = 0; g < G; ++g) s[u][g] = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack2(w[e]);
#pragma unroll
          for (int g = 0; g < G; ++g) s[u][g] += q[g][2 * e] * f.x + q[g][2 * e + 1] * f.y;
        }
      }
#pragma unroll 1
      for (int o = lpk >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int g = 0; g < G; ++g) s[u][g] += __shfl_xor_sync(0xffffffffu, s[u][g], o);
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float mn = m[g];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (j0 + u * groups > pos) s[u][g] = -INFINITY;
          mn = fmaxf(mn, s[u][g]);
        }
        const float base = mn == -INFINITY ? 0.f : mn;  // a group without keys so far
        const float corr = exp2f(m[g] - base);
        m[g] = mn;
        l[g] *= corr;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] *= corr;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          s[u][g] = exp2f(s[u][g] - base);
          l[g] += s[u][g];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t w[4] = {vr[u].x, vr[u].y, vr[u].z, vr[u].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack2(w[e]);
#pragma unroll
          for (int g = 0; g < G; ++g) {
            acc[g][2 * e] = fmaf(s[u][g], f.x, acc[g][2 * e]);
            acc[g][2 * e + 1] = fmaf(s[u][g], f.y, acc[g][2 * e + 1]);
          }
        }
      }
    }
    // groups of a warp, then the warps
#pragma unroll 1
    for (int o = lpk; o < 32; o <<= 1) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float mo = __shfl_xor_sync(0xffffffffu, m[g], o), lo = __shfl_xor_sync(0xffffffffu, l[g], o);
        const float mn = fmaxf(m[g], mo), base = mn == -INFINITY ? 0.f : mn;
        const float f = exp2f(m[g] - base), fo = exp2f(mo - base);
        m[g] = mn;
        l[g] = l[g] * f + lo * fo;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] = acc[g][e] * f + __shfl_xor_sync(0xffffffffu, acc[g][e], o) * fo;
      }
    }
    float* s_ml = sm;                    // [G][kWarps][2]
    float* s_acc = sm + G * kWarps * 2;  // [G][kWarps][hd]
    __syncthreads();                     // the previous item's merge has been read
    if (lane < lpk && act) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (sub == 0) {
          s_ml[(g * kWarps + warp) * 2] = m[g];
          s_ml[(g * kWarps + warp) * 2 + 1] = l[g];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) s_acc[(g * kWarps + warp) * a.hd + d0 + e] = acc[g][e];
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < G * a.hd / 2; i += kThreads) {
      const int g = 2 * i / a.hd, d = 2 * i - g * a.hd;
      float mx = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, s_ml[(g * kWarps + w) * 2]);
      float ls = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float f = exp2f(s_ml[(g * kWarps + w) * 2] - mx);  // warps without a key: exp2(-inf) = 0
        ls += s_ml[(g * kWarps + w) * 2 + 1] * f;
        o0 += s_acc[(g * kWarps + w) * a.hd + d] * f;
        o1 += s_acc[(g * kWarps + w) * a.hd + d + 1] * f;
      }
      const uint32_t v = pack2(o0 / ls, o1 / ls);
      const size_t at = (size_t)b * (qd / 2) + (size_t)((h0 + g) * a.hd + d) / 2;
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
  __shared__ unsigned long long s_best[32];
  __shared__ double s_before[32], s_target[32];
  __shared__ Prod s_prod[5];
  constexpr int BP = 8 * R8, J = kThreads / BP;  // a thread's row of the batch is fixed: threadIdx.x % BP
  constexpr bool kWords = R8 == 1;
  uint8_t* stage = smem;
  float2* part = reinterpret_cast<float2*>(smem + a.stage_bytes + kRingBytes);  // staged rows | ring of weights | partial sums
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
  Walk w;
  w.ring = smem_u32(smem) + (uint32_t)a.stage_bytes + (uint32_t)((warp * kSlots * 32 + lane) * 16);
  w.start(s_prod[kQkv], a.w + a.off_qkv, 0, min(a.umax, s_prod[kQkv].nu));

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
    __syncthreads();
    float bv = -INFINITY;
    int bi = -1;
    // the products of the step in order: q|k|v (then attention), Wo, W1|W3, W2 of every layer, and the classifier
#pragma unroll 1
    for (int idx = 0; idx <= 4 * a.L; ++idx) {
      const int l = idx >> 2, kind = l == a.L ? kHead : idx & 3;
      const Prod& p = s_prod[kind];
      const uint32_t epoch = (uint32_t)(step * a.L + l + 1);
      auto start_next = [&] {  // also across the end of the step: weights do not change
        const int next = idx == 4 * a.L ? 0 : idx + 1;
        const Prod& q = s_prod[next == 4 * a.L ? kHead : next & 3];
        if (step + 1 < a.n_new || idx < 4 * a.L)
          w.start(q, a.w + q.off + (size_t)(next >> 2) * q.layer_stride, 0, min(a.umax, q.nu));
      };
      if (p.nu == 0) {
        start_next();
      } else {
        const bool direct = kind == kWo || kind == kW2;
        if (!direct) {
          // x before this layer (after W2 of the one below; the embedding row for layer 0), or after Wo for W1|W3
          const bool embed = kind == kQkv && l == 0;
          const float* wn = a.p + (kind == kHead ? a.off_rms_final : (kind == kQkv ? a.off_rms_att : a.off_rms_ffn) + (size_t)l * a.rms_stride);
          if (kWords && !embed) {
            const uint2* x = kind == kW13 ? a.w_x1 : a.w_x0;
            stage_norm<R8, true>(D, a.B, [&](int r) { return x + (size_t)r * D; }, kind == kW13 ? epoch : epoch - 1, wn, stage, wait);
          } else {
            stage_norm<R8, false>(D, a.B, [&](int r) { return embed ? a.p + a.off_embed_f32 + (size_t)s_tok[r] * D : a.x + (size_t)r * D; },
                                  0u, wn, stage, wait);
          }
          __syncthreads();
        } else if (kWords) {
          __syncthreads();  // the partial sums of the phase before have been read
        }
#pragma unroll 1
        for (int g0 = 0; g0 < p.nu; g0 += a.umax) {
          const int n = min(a.umax, p.nu - g0);
          if (!direct) {
            run_product<R8>(p, w, n, part, StagedRows<R8>{reinterpret_cast<const uint4*>(stage)});
          } else if constexpr (kWords) {
            run_product<R8>(p, w, n, part, WordRows{kind == kWo ? a.w_att : a.w_gate, a.B, epoch, wait});
          } else {
            run_product<R8>(p, w, n, part, PlainRows<R8>{kind == kWo ? a.att : a.gate, a.B});
          }
          if (g0 + n < p.nu) w.start(p, a.w + p.off + (size_t)l * p.layer_stride, g0 + n, min(a.umax, p.nu - g0 - n));
          else start_next();
          __syncthreads();
          if (live) {
            if (kind == kW13) {
#pragma unroll 1
              for (int i = j0; i < n * 2; i += J) {
                const int u = (i >> 2) * 2, c = i & 3;
                const float2 h1 = pair_sum<R8>(part, u, row, c), h3 = pair_sum<R8>(part, u + 1, row, c);
                const uint32_t g = pack2(h1.x * h3.x * sigmoid(h1.x), h1.y * h3.y * sigmoid(h1.y));
                const int pair = (int)blockIdx.x + ((g0 + u) >> 1) * (int)gridDim.x;
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
                    const int r = pos * (a.hd / 2) + (col % a.hd) / 2;
                    const float c = a.cosb[r], sn = a.sinb[r];
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
                  float2 old;
                  if (kind == kWo && l == 0) {
                    old = __ldg(reinterpret_cast<const float2*>(a.p + a.off_embed_f32 + (size_t)s_tok[row] * D + col));
                  } else if (kWords) {
                    const uint4 o = get_words((kind == kWo ? a.w_x0 : a.w_x1) + at);  // complete: this CTA has staged it
                    old = make_float2(__uint_as_float(o.x), __uint_as_float(o.z));
                  } else {
                    old = __ldcg(reinterpret_cast<const float2*>(a.x + at));
                  }
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
      if (kWords) {
        if (s_abort) return;
      } else if (kind != kHead && !bar.sync()) {
        return;
      }
      if (kind == kQkv) {
        const size_t cl = (size_t)l * a.kv_layer;
        float* sm = reinterpret_cast<float*>(part);
        if (a.group == 3) attention_phase<R8, 3>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
        else if (a.group == 2) attention_phase<R8, 2>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
        else attention_phase<R8, 1>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
        if (!kWords && !bar.sync()) return;
      }
    }
    // ---- the best logit of every row
    if (bi >= 0) atomicMax(&s_best[row], pack_best(bv, bi));
    __syncthreads();
    if ((int)threadIdx.x < a.B && s_best[threadIdx.x] != 0) atomicMax(best + threadIdx.x, s_best[threadIdx.x]);
    if (!bar.sync()) return;
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
    if (!bar.sync()) return;
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
    if (!bar.sync()) return;
  }
  if (!sampling && a.n_new > 1 && blockIdx.x == 0 && (int)threadIdx.x < a.B) {
    const unsigned long long k = __ldcg(a.best + ((a.n_new - 1) % 3) * a.B + threadIdx.x);
    a.out[(size_t)threadIdx.x * a.n_new + a.n_new - 1] = (uint16_t)(k == 0 ? 0 : 0xffffffffu - (uint32_t)k);
  }
}

size_t stage_bytes(int r8, int D) { return (size_t)((D + 31) / 32) * r8 * 512; }
size_t unit_bytes(int r8) { return sizeof(float2) * kWarps * (size_t)(r8 == 1 ? Part<1>::kVecs : r8 == 2 ? Part<2>::kVecs : Part<4>::kVecs); }
constexpr size_t kSmemLimit = 222 * 1024;  // beside the static arrays

// Units per group: as many as shared memory holds beside the staged activations (a power of two, 2..32; W1|W3 units
// come in pairs).
int decode_umax(int r8, int D) {
  for (int u = 32; u >= 2; u >>= 1)
    if (stage_bytes(r8, D) + kRingBytes + u * unit_bytes(r8) <= kSmemLimit) return u;
  return 0;
}
int row_groups(int batch) { return batch <= 8 ? 1 : batch <= 16 ? 2 : 4; }

}  // namespace

bool decode_steps_supported(int D, int Hd, int H, int KV, int hd, int V, int batch) {
  return batch >= 1 && batch <= 32 && hd % 8 == 0 && hd <= 128 && D % 8 == 0 && Hd % 32 == 0 && V % 8 == 0 && H % KV == 0 &&
         decode_umax(row_groups(batch), D) > 0;
}
size_t decode_words_bytes(int D, int Hd, int H, int KV, int hd) {  // exchange buffers of up to 8 sequences
  return sizeof(uint2) * 8 * ((size_t)2 * D + (size_t)(H + 2 * KV) * hd / 2 + (size_t)H * hd / 2 + (size_t)Hd / 2);
}

int decode_steps(DecodeArgs a, void* words, int sms, cudaStream_t s) {
  if (a.n_new < 2) return 0;
  const int r8 = row_groups(a.B), qd = a.H * a.hd, qkv = (a.H + 2 * a.KV) * a.hd;
  a.umax = decode_umax(r8, a.D);
  if (a.umax == 0) return -2;
  a.stage_bytes = (int)stage_bytes(r8, a.D);
  // The exchange of flagged words needs every CTA to own units of q|k|v and of W1|W3; more CTAs than that would idle anyway.
  const int ctas = std::min(sms, std::min(qkv / 8, a.Hd / 8));
  // Query heads per attention item: heads that share keys read them once, as long as the items still fill half of the
  // SMs; a single sequence takes one head per CTA.
  const int rep = a.H / a.KV;
  a.group = 1;
  for (int g = 3; g > 1; --g)
    if (rep % g == 0 && a.B * (a.H / g) * 2 >= ctas) {
      a.group = g;
      break;
    }
  uint2* p = reinterpret_cast<uint2*>(words);
  a.w_x0 = p; p += (size_t)8 * a.D;
  a.w_x1 = p; p += (size_t)8 * a.D;
  a.w_qkv = p; p += (size_t)8 * qkv / 2;
  a.w_att = p; p += (size_t)8 * qd / 2;
  a.w_gate = p;
  // the attention merge and the sampler's sums use the partial sums' memory
  size_t tail = a.umax * unit_bytes(r8);
  tail = std::max(tail, sizeof(float) * (size_t)(3 * kWarps * (2 + a.hd)));
  tail = std::max(tail, sizeof(double) * (size_t)ctas * a.B);
  const size_t bytes = a.stage_bytes + kRingBytes + tail;
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
