// KV-cached generation for up to 8 sequences: all steps after the prefill in ONE persistent cooperative kernel (llama-style
// architecture, bf16 engines).  (decode_batch.cu: more sequences, and wider models.)
//
// A decode step is about sixty dependent products with a few rows.  Launched one by one each of them costs the
// fixed latency of a kernel (a 128-row tensor-core tile of the training GEMM takes 10-15 us for 8 KB of useful output),
// although the bytes of a step -- every weight once, keys and values once -- take 35 us at the memory's rate.  Here
// one CTA per SM stays resident and walks through the five phases of a layer (q|k|v, attention, Wo, W1|W3, W2).  What
// bounds it is the latency of a phase: how fast one SM's results reach all others, and the chain of instructions
// between reading activations and publishing results.  So:
//   * Weights never change, and the 8 weight rows of a unit are one contiguous piece of 16 K bytes: one thread streams
//     them into a ring of shared-memory slots with bulk copies, as far ahead as the ring reaches, across phases and steps.
//     (Measured with all SMs reading: 30 B/clk per SM through per-lane loads or cp.async, 70 through bulk copies.)
//   * Results are exchanged as 8-byte words {value, epoch}, written and read with single 64-bit accesses.  A reader polls
//     the words it needs; there is no barrier, no fence and no second round trip (a grid barrier with its stores and
//     loads takes 1.8 us on this GPU, a flagged word about 0.6).
//   * All products run through one copy of the code (staging, MMA loop, reduction), so it stays in the instruction cache.
//
// Products: y[b, n] = sum_k x[b, k] W[n, k] with mma.sync m16n8k16 -- the sequences are the A rows (8 of 16 used), 8
// weight rows the B columns, so a "unit" of work is 8 weight rows and N / 8 units deal out evenly over the
// SMs.  tcgen05 tiles start at 64 rows of A and would leave most of the tile empty.  Inside a CTA the sixteen warps split
// the contraction in 32-wide chunks (a warp's A fragments then stay in registers for all units of the CTA) and their
// partial sums meet in shared memory.  The order of k inside a chunk is free as long as both operands agree, so every
// lane reads 16 contiguous bytes of a weight row (k = 8 (lane % 4) ..) and uses them as the fragments of two MMAs: no
// ldmatrix.
#include <algorithm>
#include <cmath>

#include "decode_common.cuh"

namespace ane {
namespace {

constexpr int kWarps = 16, kThreads = kWarps * 32, kRows = 8;

// One unit's partial sums of one slice of the contraction: float2 [4 column pairs][8 rows], pitch free of bank conflicts.
constexpr int kPitch = 12, kVecs = 4 * kPitch;

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
constexpr int kUnits = 4, kSlots = 3;  // units per group (even, because W1|W3 units come in pairs); slots
struct Feed {
  uint32_t bar, slot;  // shared-memory addresses of the first barrier and slot
  int slot_bytes, issued, used;
  int step, idx, g0;   // next group
  __device__ __forceinline__ void issue(const DecodeArgs& a, const Prod* prods) {
#pragma unroll 1
    while (issued - used < kSlots && step < a.n_new) {
      const int layer = idx >> 2;
      const Prod& p = prods[layer == a.L ? kHead : idx & 3];
      const int n = min(kUnits, p.nu - g0);
      if (n > 0) {
        const int at = issued % kSlots;
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
  const uint4* stage;  // nullptr: words
  const uint2* words;  // {two values, epoch}
  int B;
  uint32_t epoch;
};
__device__ __forceinline__ void read_a(uint4 (&f)[4], const Source& s, const Share& w, int first, const Wait& wait) {
  const int lane = threadIdx.x & 31, g = lane >> 2, left = w.nc - first;
  if (s.stage != nullptr) {
    const uint4* st = s.stage + (size_t)(w.c0 + first) * 32 + lane;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < left) f[c] = st[c * 32];
    return;
  }
  const int k = (w.c0 + first) * 32 + (lane & 3) * 8;
  const uint2* p = s.words + ((size_t)(g < s.B ? g : 0) * w.K + k) / 2;
  long long t0 = 0;
#pragma unroll 1
  for (unsigned n = 0;; ++n) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool take = c < left && k + c * 32 < w.K && g < s.B;
      const uint4 x = get_words_if(p + c * 16, take, s.epoch), y = get_words_if(p + c * 16 + 2, take, s.epoch);
      ok = ok && words_are(x, s.epoch) && words_are(y, s.epoch);
      f[c] = make_uint4(x.x, x.z, y.x, y.z);
    }
    if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) return;
  }
}

// Partial sums of the n units in a slot (rows of K bf16): this warp's chunks.
__device__ __forceinline__ void run_units(const Share& w, int n, const uint8_t* slot, float2* part, const Source& src, uint4 (&a)[4], bool read, const Wait& wait) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* d = part + (size_t)warp * kVecs + (lane & 3) * kPitch + (lane >> 2);
  const int k0 = w.c0 * 32 + (lane & 3) * 8;
  const uint4* wp = reinterpret_cast<const uint4*>(slot) + ((lane >> 2) * w.K + k0) / 8;
#pragma unroll 1
  for (; n > 0; --n) {
    float acc0 = 0.f, acc1 = 0.f;
#pragma unroll 1
    for (int blk = 0; blk == 0 || blk < w.nc; blk += 4) {
      if (read) read_a(a, src, w, blk, wait);
      read = w.nc > 4;  // four chunks or fewer: the same fragments for every unit
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (blk + c < w.nc) {
          uint4 b = make_uint4(0, 0, 0, 0);
          if (k0 + (blk + c) * 32 < w.K) b = wp[(blk + c) * 4];
          mma16816_top(acc0, acc1, a[c].x, a[c].y, b.x, b.y);
          mma16816_top(acc0, acc1, a[c].z, a[c].w, b.z, b.w);
        }
      }
    }
    *d = make_float2(acc0, acc1);
    d += kWarps * kVecs;
    wp += w.K;
  }
}

// Sum over the warps of column pair (2c, 2c + 1) of row b.
__device__ __forceinline__ float2 pair_sum(const float2* part, int unit, int b, int c) {
  const float2* d = part + (size_t)unit * kWarps * kVecs + c * kPitch + b;
  float2 s = make_float2(0.f, 0.f), t = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kWarps; i += 2) {
    const float2 u = d[i * kVecs], v = d[(i + 1) * kVecs];
    s.x += u.x;
    s.y += u.y;
    t.x += v.x;
    t.y += v.y;
  }
  return make_float2(s.x + t.x, s.y + t.y);
}

// ---- activations into A fragments -------------------------------------------------------------------------------------
// stage[chunk][lane]: byte offset of element k of row r.  Rows past the batch stay zero from the start.
__device__ __forceinline__ int frag_at(int r, int k) { return (((k >> 5) * 32 + r * 4 + ((k & 31) >> 3)) << 4) + (k & 7) * 2; }

// Which row a warp normalises: the sequences share the warps, 16 / B per row.
struct RowShare {
  int row, sub, per_row;
};
// Normalised rows, bf16(x * rms^-1 * gain), rounded like the training forward's.  row(r) = plain fp32 values; words:
// {value, epoch} pairs instead.  A warp's part of a row stays in registers between the sum of squares and the
// conversion; rows wider than that go through in segments and are read twice.  gains: the norm's weights in shared memory.
template <class Row>
__device__ __forceinline__ void stage_norm(int K, int B, Row row, const uint2* words, uint32_t epoch, const float* gains, uint8_t* stage,
                                           float* s_sq, const RowShare& sh, float inv_dim, const Wait& wait) {
  constexpr int V = 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = sh.row;
  const int stride = sh.per_row * 128, seg = stride * V, nseg = (K + seg - 1) / seg;
  const bool has = r < B;
  const float* px = row(has ? r : 0);
  const uint2* pw = words + (size_t)(has ? r : 0) * K;
  float sq = 0.f, rms = 0.f;
#pragma unroll 1
  for (int it = 0; it < (nseg == 1 ? 1 : 2 * nseg); ++it) {
    const int k0 = (it < nseg ? it : it - nseg) * seg + (sh.sub * 32 + lane) * 4;
    float4 x[V];
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = ldf_l2_if(px + k0 + i * stride, has && k0 + i * stride < K && words == nullptr);
    if (words != nullptr) {
      long long t0 = 0;
#pragma unroll 1
      for (unsigned n = 0;; ++n) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const bool take = has && k0 + i * stride < K;
          const uint4 a = get_words_if(pw + k0 + i * stride, take, epoch), b = get_words_if(pw + k0 + i * stride + 2, take, epoch);
          ok = ok && words_are(a, epoch) && words_are(b, epoch);
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
      if (lane == 0) s_sq[warp] = sq;
      __syncthreads();
      sq = 0.f;  // the row's other warps
#pragma unroll 1
      for (int i = 0; i < sh.per_row; ++i) sq += s_sq[warp - sh.sub + i];
      rms = inverse_sqrt(fmaf(sq, inv_dim, 1e-5f));
    }
    if (it >= nseg || nseg == 1) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        if (!has || k0 + i * stride >= K) continue;
        const float4 g = *reinterpret_cast<const float4*>(gains + k0 + i * stride);
        *reinterpret_cast<uint2*>(stage + frag_at(r, k0 + i * stride)) =
            make_uint2(pack2(x[i].x * rms * g.x, x[i].y * rms * g.y), pack2(x[i].z * rms * g.z, x[i].w * rms * g.w));
      }
    }
  }
}

// PANELS: 64 dims of a head each (one kernel for both spilled the shorter heads' registers as well).
template <int PANELS>
__global__ void __launch_bounds__(kThreads, 1) decode_steps_kernel(const __grid_constant__ DecodeArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_tok[32], s_abort;
  __shared__ float s_sq[2 * kWarps], s_cos[64], s_sin[64];
  __shared__ __align__(8) uint64_t s_full[kSlots];
  __shared__ unsigned long long s_best[32];
  __shared__ double s_before[32], s_target[32];
  __shared__ Prod s_prod[5];
  constexpr int J = kThreads / kRows;  // a thread's row of the batch is fixed: threadIdx.x % 8
  uint8_t* stage = smem;
  float2* part = reinterpret_cast<float2*>(smem + a.stage_bytes + kSlots * a.slot_bytes);  // staged rows | ring of weights | partial sums
  const int row = threadIdx.x % kRows, j0 = threadIdx.x / kRows;
  const int warp = threadIdx.x >> 5;
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
  share.per_row = kWarps / a.B;
  share.row = warp / share.per_row;
  share.sub = warp - share.row * share.per_row;
  constexpr int kFeeder = kThreads - 32;
  Feed feed{smem_u32(s_full), smem_u32(smem) + (uint32_t)a.stage_bytes, a.slot_bytes, 0, 0, 1, 0, 0};
  if (threadIdx.x == kFeeder) {
    for (int i = 0; i < kSlots; ++i) mbar_init(feed.bar + 8u * i, 1);
    fence_mbar_init();
    feed.issue(a, s_prod);
  }
  __syncthreads();
  int group = 0;  // groups consumed
  auto group_ready = [&] {
    if (!mbar_wait(feed.bar + 8u * (group % kSlots), (uint32_t)(group / kSlots) & 1u, a.status, DEV_GRID_TIMEOUT)) s_abort = 1;
  };
  // every way out before the end: no copy may still be on its way into this CTA's shared memory
  auto leave = [&] {
    if (threadIdx.x == kFeeder)
      for (int i = feed.used; i < feed.issued; ++i)
        mbar_wait(feed.bar + 8u * (i % kSlots), (uint32_t)(i / kSlots) & 1u, nullptr, 0);
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
      Source src{nullptr, nullptr, a.B, epoch};
      float2 old = make_float2(0.f, 0.f);  // residual of this thread's first pair
      const uint2* wrow = (kind == kWo ? a.w_x0 : a.w_x1) + (size_t)row * D;
      auto residual = [&](int col) {
        if (kind == kWo && l == 0) return __ldg(reinterpret_cast<const float2*>(a.p + a.off_embed_f32 + (size_t)s_tok[live ? row : 0] * D + col));
        const uint4 o = get_words(wrow + col);  // complete: this CTA has staged it
        return make_float2(__uint_as_float(o.x), __uint_as_float(o.z));
      };
      if (direct) {
        __syncthreads();  // the partial sums of the phase before have been read
        src.words = kind == kWo ? a.w_att : a.w_gate;
        if (live && j0 < p.nu * 4) old = residual(p.row0(j0 >> 2) + 2 * (j0 & 3));
      } else if (p.nu > 0) {  // (a CTA beyond the units of a small vocabulary has no group to wait for)
        // x before this layer (after W2 of the one below; the embedding row for layer 0), or after Wo for W1|W3
        const bool embed = kind == kQkv && l == 0;
        const uint2* words = embed ? nullptr : kind == kW13 ? a.w_x1 : a.w_x0;
        group_ready();
        const float* gains = reinterpret_cast<const float*>(smem + a.stage_bytes + (group % kSlots + 1) * a.slot_bytes - D * 4);
        stage_norm(D, a.B, [&](int r) { return a.p + a.off_embed_f32 + (size_t)(embed ? s_tok[r] : 0) * D; }, words,
                       kind == kW13 ? epoch : epoch - 1, gains, stage, s_sq, share, a.inv_dim, wait);
        __syncthreads();
        src.stage = reinterpret_cast<const uint4*>(stage);
      }
      {
        const Share mine = make_share(p.K);
        uint4 frag[4] = {};  // (defined on every path: not live from one product to the next)
#pragma unroll 1
        for (int g0 = 0; g0 < p.nu; g0 += kUnits, ++group) {
          const int n = min(kUnits, p.nu - g0);
          group_ready();
          run_units(mine, n, smem + a.stage_bytes + (group % kSlots) * a.slot_bytes, part, src, frag, g0 == 0, wait);
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
                const float2 h1 = pair_sum(part, u, row, c), h3 = pair_sum(part, u + 1, row, c);
                const uint32_t g = pack2(h1.x * h3.x * sigmoid(h1.x), h1.y * h3.y * sigmoid(h1.y));
                const int pair = (int)blockIdx.x + ((g0 + u) >> 1) * (int)gridDim.x;  // columns 8 pair .. of the gate
                const size_t at = (size_t)row * (a.Hd / 2) + pair * 4 + c;
                put_word(a.w_gate + at, g, epoch);
              }
            } else {
#pragma unroll 1
              for (int i = j0; i < n * 4; i += J) {
                const float2 s = pair_sum(part, i >> 2, row, i & 3);
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
                  put_word(a.w_qkv + (size_t)row * ((QD + 2 * KVD) / 2) + col / 2, v, epoch);
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
                  uint2* to = (kind == kWo ? a.w_x1 : a.w_x0) + at;
                  put_word(to, __float_as_uint(x), epoch);
                  put_word(to + 1, __float_as_uint(y), epoch);
                }
              }
            }
          }
          if (g0 + n < p.nu) __syncthreads();
        }
      }
      if (s_abort != 0) {
        leave();
        return;
      }
      if (kind == kQkv) {
        const size_t cl = (size_t)l * a.kv_layer;
        float* sm = reinterpret_cast<float*>(part);
        attention_phase<PANELS, kWarps, 1>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
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
    if (sampling && !sample_tokens<kWarps>(a, step, best, reinterpret_cast<double*>(part), s_tok, s_before, s_target, [&] { return bar.sync(); })) {
      leave();
      return;
    }
  }
  if (!sampling && a.n_new > 1 && blockIdx.x == 0 && (int)threadIdx.x < a.B) {
    const unsigned long long k = __ldcg(a.best + ((a.n_new - 1) % 3) * a.B + threadIdx.x);
    a.out[(size_t)threadIdx.x * a.n_new + a.n_new - 1] = (uint16_t)(k == 0 ? 0 : 0xffffffffu - (uint32_t)k);
  }
}

size_t stage_bytes(int D) { return (size_t)((D + 31) / 32) * 512; }
// a group's units with the norm's gains behind them, or the W2 units of a CTA (mostly one)
size_t slot_bytes(int D, int Hd, int ctas) {
  const int w2 = std::min(kUnits, (D / 8 + ctas - 1) / ctas);
  return std::max((size_t)16 * w2 * Hd, (size_t)16 * kUnits * D + 4 * D);
}
size_t tail_bytes(int hd, int ctas, int B) {  // partial sums; the attention merge and the sampler's sums use the same memory
  return std::max(sizeof(float2) * kWarps * kVecs * kUnits,
                  std::max(sizeof(float) * (size_t)(kWarps * 8 * (2 + (hd <= 64 ? 64 : 128))), sizeof(double) * (size_t)ctas * B));
}
size_t smem_bytes(int D, int Hd, int hd, int ctas, int B) { return stage_bytes(D) + kSlots * slot_bytes(D, Hd, ctas) + tail_bytes(hd, ctas, B); }
constexpr size_t kSmemLimit = 224 * 1024;  // beside the static arrays

// The exchange of flagged words needs every CTA to own units of q|k|v and of W1|W3; more CTAs than that would idle anyway.
// A multiple of 4: see Prod.
int decode_ctas(int sms, int Hd, int H, int KV, int hd) { return std::min(std::min(sms, 148), std::min((H + 2 * KV) * hd / 8, Hd / 8)) & ~3; }

// Up to 8 sequences go to the kernel above where its whole rows fit (dim <= 1100 or so): one SM's part of a contraction costs
// it little then, and nothing has to be exchanged in a cluster.  Prompts of 37 tokens and 64 new ones, this kernel against
// clusters, for 1 / 4 / 8 sequences: 13.2 / 13.6 / 14.6 against 18.6 / 18.8 / 19.2 ms (110M model), 8.5 / 8.6 / 8.9 against
// 11.9 / 12.0 / 12.1 (dim 512), 6.7 / 6.5 / 6.6 against 8.2 / 8.4 / 8.5 (dim 288); with prompts of 512 and with grouped heads
// alike.  The others take the clusters.
bool in_clusters(int D, int Hd, int H, int KV, int hd, int batch, int sms) {
  const int ctas = decode_ctas(sms, Hd, H, KV, hd);
  return batch > kRows || ctas <= 0 || smem_bytes(D, Hd, hd, ctas, batch) > kSmemLimit;
}
size_t word_rows(int D, int Hd, int H, int KV, int hd, int batch, int sms) { return in_clusters(D, Hd, H, KV, hd, batch, sms) ? 32 : kRows; }

}  // namespace

bool decode_steps_supported(int D, int Hd, int H, int KV, int hd, int V, int batch, int sms) {
  return batch >= 1 && batch <= 32 && hd % 8 == 0 && hd <= 128 && D % 8 == 0 && H * hd == D && Hd % 32 == 0 && V % 8 == 0 && H % KV == 0 &&
         (!in_clusters(D, Hd, H, KV, hd, batch, sms) || decode_batch_supported(D, Hd, hd, batch, sms));
}
size_t decode_words_bytes(int D, int Hd, int H, int KV, int hd, int batch, int sms) {
  return sizeof(uint2) * word_rows(D, Hd, H, KV, hd, batch, sms) * ((size_t)2 * D + (size_t)(H + 2 * KV) * hd / 2 + (size_t)H * hd / 2 + (size_t)Hd / 2);
}

int decode_steps(DecodeArgs a, void* words, int sms, cudaStream_t s) {
  if (a.n_new < 2) return 0;
  const int qd = a.H * a.hd, qkv = (a.H + 2 * a.KV) * a.hd;
  const int rep = a.H / a.KV;
  a.group = rep <= 8 ? rep : 1;  // query heads per attention item: rows of one fragment
  a.rep = rep;
  a.items = a.H / a.group;
  a.hd_magic = quotient_magic((unsigned)a.hd);
  a.rep_magic = quotient_magic((unsigned)a.rep);
  a.items_magic = quotient_magic((unsigned)a.items);
  a.score_scale = 1.4426950408889634f / sqrtf((float)a.hd);
  a.inv_dim = 1.0f / (float)a.D;
  const size_t rows = word_rows(a.D, a.Hd, a.H, a.KV, a.hd, a.B, sms);
  uint2* p = reinterpret_cast<uint2*>(words);
  a.w_x0 = p; p += rows * a.D;
  a.w_x1 = p; p += rows * a.D;
  a.w_qkv = p; p += rows * qkv / 2;
  a.w_att = p; p += rows * qd / 2;
  a.w_gate = p;
  if (cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s) != cudaSuccess ||
      cudaMemsetAsync(words, 0, decode_words_bytes(a.D, a.Hd, a.H, a.KV, a.hd, a.B, sms), s) != cudaSuccess ||
      cudaMemsetAsync(a.best, 0, 3 * sizeof(unsigned long long) * (size_t)a.B, s) != cudaSuccess)
    return -3;
  if (in_clusters(a.D, a.Hd, a.H, a.KV, a.hd, a.B, sms)) return decode_batch_steps(a, sms, s);
  const int ctas = decode_ctas(sms, a.Hd, a.H, a.KV, a.hd);
  a.stage_bytes = (int)stage_bytes(a.D);
  a.slot_bytes = (int)slot_bytes(a.D, a.Hd, ctas);
  const size_t bytes = smem_bytes(a.D, a.Hd, a.hd, ctas, a.B);
  auto kern = a.hd <= 64 ? decode_steps_kernel<1> : decode_steps_kernel<2>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return -3;
  void* args[] = {&a};
  // cooperative: all CTAs are resident together, so the waits on one another complete
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(ctas), dim3(kThreads), args, bytes, s) == cudaSuccess ? 0 : -4;
}

}  // namespace ane
