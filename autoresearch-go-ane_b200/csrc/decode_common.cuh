// Pieces shared by the two persistent decode kernels: decode.cu (up to 8 sequences, results exchanged as flagged words)
// and decode_batch.cu (9 to 32, clusters that split every contraction).
#pragma once
#include "common.cuh"
#include "decode_math.h"
#include "kernels.h"

namespace ane {
namespace {

// Barrier of the NW warps that compute (a kernel may have one more that only copies).
template <int NW>
__device__ __forceinline__ void cta_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
}
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

// 1 / x for divide(), |x| up to 2^126.  1 / sqrt(x).
__device__ __forceinline__ float inverse(float x) { return newton_inverse(x, __fdividef(1.0f, x)); }
__device__ __forceinline__ float inverse_sqrt(float x) { return newton_inverse_sqrt(x, rsqrtf(x)); }
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

// ---- exchange of results between SMs ---------------------------------------------------------------------------------
// Word buffers: x0 (stream after W2), x1 (after Wo), q|k|v, attention out, gate; epoch = step * layers + layer + 1.
// Why a word is never overwritten while someone still needs it: every CTA, or cluster, owns units of q|k|v and of W1|W3 (the
// grid is cut down for that).  x1 of the next layer is written by one that has read all heads' attention outputs, hence all
// q|k|v units of that layer, and each owner produced its own only after it had read all of x1.  In the same way x0 follows
// all gates, hence everybody's W1|W3 units; gates, attention outputs and q|k|v words follow a complete x1, x0 and x0, whose
// owners had read them.
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

// The same where `take`, else {0, other, 0, other}; in one instruction, so that a run of them is in flight together.
__device__ __forceinline__ uint4 get_words_if(const uint2* p, bool take, uint32_t other) {
  const unsigned long long none = (unsigned long long)other << 32;
  unsigned long long a = none, b = none;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n\t}"
               : "+l"(a), "+l"(b) : "l"(p), "r"((uint32_t)take) : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ bool words_are(uint4 w, uint32_t epoch) { return w.y == epoch && w.w == epoch; }

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

// ---- attention ------------------------------------------------------------------------------------------------------
// One new token per sequence over cache positions 0..pos.  A work item is one sequence and the (up to 8) query heads
// of one KV head; every warp takes 16 keys at a time and keeps a running maximum, sum and P*V, merged at the end.  No
// operand is transposed or staged:
//   scores  A = q (rows are heads), B[k = dim, n = key]: lane (g, c) reads 16 bytes of key g at dims 8c.. and 32 + 8c..,
//           two MMAs each (the order of k is free as long as q is read the same way);
//   P * V   A[row, k = key] = V transposed, B = P: lane (g, c) reads dims 8g.. of keys 2c, 2c + 1, 2c + 8, 2c + 9; MMA j
//           takes elements 2j and 2j + 1 of each, so its rows g and g + 8 stand for dims 8g + 2j and 8g + 2j + 1.  (P as A
//           would leave 8 of 16 rows empty.)  P enters as bf16 hi + lo, two MMAs, so that it keeps 16 bits.
// hd <= 64 is one panel of 64 dims (what lies past hd reads as zero), up to 128 two.  q and the new key and
// value come from flagged words, the older ones from the cache.  U tiles of 16 keys per warp are in flight: the
// loads of a tile are issued again as soon as its MMAs have read the registers, and the first ones (the cache does not
// depend on q) before q is there.
template <int PANELS, int NW, int U>
__device__ __forceinline__ void attention_phase(const DecodeArgs& a, const bf16* kc, const bf16* vc, int pos, float* sm, uint32_t epoch, const Wait& wait) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  // opaque: what follows from the sizes is computed here, not kept in registers (or spilled) through the whole generation
  int hd = a.hd, G = a.group, H = a.H, KV = a.KV;
  asm volatile("" : "+r"(hd), "+r"(G), "+r"(H), "+r"(KV));
  const int kvd = KV * hd, qd = H * hd, hgroups = a.items;
  const float sc = a.score_scale;  // scores in the log2 domain
  constexpr int kStep = NW * 16;                              // keys of one tile of every warp
#pragma unroll 1
  for (int item = blockIdx.x; item < a.B * hgroups; item += gridDim.x) {
    const int b = quotient(item, hgroups, a.items_magic), h0 = (item - b * hgroups) * G, kvh = quotient(h0, a.rep, a.rep_magic);
    const bf16* kb = kc + (size_t)b * a.S * kvd + (size_t)kvh * hd;
    const bf16* vb = vc + (size_t)b * a.S * kvd + (size_t)kvh * hd;
    const uint2* wk = nullptr;  // words of the new key
    // 16 bytes of a key's or value's dims d..d+7 from the cache: all but the newest, which put_new() adds
    uint4 kr[U][2][2 * PANELS], vr[U][4][PANELS];
    auto fetch = [&](const bf16* base, int j, int d) { return ld_l2_if(base + (size_t)j * kvd + d, d < hd && j < pos); };
    auto load_k = [&](int u, int j0) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int i = 0; i < 2 * PANELS; ++i) kr[u][t][i] = fetch(kb, j0 + t * 8 + g, i * 32 + c * 8);
    };
    auto load_v = [&](int u, int j0) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int p = 0; p < PANELS; ++p) vr[u][t][p] = fetch(vb, j0 + 2 * c + (t & 1) + (t >> 1) * 8, p * 64 + g * 8);
    };
#pragma unroll
    for (int u = 0; u < U; ++u) {
      load_k(u, warp * 16 + u * kStep);
      load_v(u, warp * 16 + u * kStep);
    }
    uint4 q[PANELS][2];
    const uint2* row = a.w_qkv + (size_t)b * ((qd + 2 * kvd) / 2);
    wk = row + (qd + kvh * hd) / 2;
    // every word of this item: q rows, key and value (the last two are read again below, from L2 as well)
    long long t0 = 0;
#pragma unroll 1
    for (unsigned n = 0;; ++n) {
      bool ok = true;
#pragma unroll
      for (int i = 0; i < 2 * PANELS; ++i) {
        const int d = i * 32 + c * 8;
        q[i >> 1][i & 1] = make_uint4(0, 0, 0, 0);
        if (d < hd) {
          const uint4 k0 = get_words(wk + d / 2), k1 = get_words(wk + d / 2 + 2), v0 = get_words(wk + (kvd + d) / 2), v1 = get_words(wk + (kvd + d) / 2 + 2);
          ok = ok && k0.y == epoch && k0.w == epoch && k1.y == epoch && k1.w == epoch && v0.y == epoch && v0.w == epoch && v1.y == epoch && v1.w == epoch;
          if (g < G) {
            const uint2* p = row + ((h0 + g) * hd + d) / 2;
            const uint4 x = get_words(p), y = get_words(p + 2);
            ok = ok && x.y == epoch && x.w == epoch && y.y == epoch && y.w == epoch;
            q[i >> 1][i & 1] = make_uint4(x.x, x.z, y.x, y.z);
          }
        }
      }
      if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
    }
    auto put_new = [&](uint4& v, int off, int j, int d) {
      if (j == pos && d < hd) {
        const uint4 x = get_words(wk + (off + d) / 2), y = get_words(wk + (off + d) / 2 + 2);
        v = make_uint4(x.x, x.z, y.x, y.z);
      }
    };
    float m = -INFINITY, l = 0.f, acc[PANELS][4][4] = {};
#pragma unroll 1
    for (int base = warp * 16; base <= pos; base += U * kStep) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j0 = base + u * kStep;
        if (j0 > pos) break;
        if (j0 + 16 > pos) {  // this warp holds the newest key
#pragma unroll
          for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < 2 * PANELS; ++i) put_new(kr[u][t][i], 0, j0 + t * 8 + g, i * 32 + c * 8);
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int p = 0; p < PANELS; ++p) put_new(vr[u][t][p], kvd, j0 + 2 * c + (t & 1) + (t >> 1) * 8, p * 64 + g * 8);
        }
        float s[2][2] = {}, mn = m;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
#pragma unroll
          for (int i = 0; i < 2 * PANELS; ++i) {
            const uint4 k = kr[u][t][i], x = q[i >> 1][i & 1];
            mma16816_top(s[t][0], s[t][1], x.x, x.y, k.x, k.y);
            mma16816_top(s[t][0], s[t][1], x.z, x.w, k.z, k.w);
          }
        }
        load_k(u, j0 + U * kStep);
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
        const float corr0 = __shfl_sync(0xffffffffu, corr, 8 * c), corr1 = __shfl_sync(0xffffffffu, corr, 8 * c + 4);  // heads 2c, 2c + 1
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
          const uint4 *v0 = &vr[u][0][p], *v1 = &vr[u][1][p], *v2 = &vr[u][2][p], *v3 = &vr[u][3][p];
          const uint32_t x[4][4] = {{v0->x, v1->x, v2->x, v3->x}, {v0->y, v1->y, v2->y, v3->y}, {v0->z, v1->z, v2->z, v3->z}, {v0->w, v1->w, v2->w, v3->w}};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float* d = acc[p][j];
            d[0] *= corr0; d[1] *= corr1; d[2] *= corr0; d[3] *= corr1;
            const uint32_t a0 = __byte_perm(x[j][0], x[j][1], 0x5410u), a1 = __byte_perm(x[j][0], x[j][1], 0x7632u);
            const uint32_t a2 = __byte_perm(x[j][2], x[j][3], 0x5410u), a3 = __byte_perm(x[j][2], x[j][3], 0x7632u);
            mma16816(d, a0, a1, a2, a3, hi[0], hi[1]);
            mma16816(d, a0, a1, a2, a3, lo[0], lo[1]);
          }
        }
        load_v(u, j0 + U * kStep);
      }
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    constexpr int kPitch = PANELS * 64 + 2;  // per warp and head: P*V, maximum, sum
    float* mine = sm + warp * 8 * kPitch;
    cta_sync<NW>();                         // the previous item's merge has been read
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (2 * c + e >= G) continue;
#pragma unroll
      for (int p = 0; p < PANELS; ++p)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<float2*>(mine + (2 * c + e) * kPitch + p * 64 + 8 * g + 2 * j) = make_float2(acc[p][j][e], acc[p][j][2 + e]);
    }
    if (g < G && c == 0) *reinterpret_cast<float2*>(mine + g * kPitch + PANELS * 64) = make_float2(m, l);
    cta_sync<NW>();
    const int used = min(NW, pos / 16 + 1);  // warps that had keys
#pragma unroll 1
    for (int i = threadIdx.x; i < G * hd / 2; i += NW * 32) {
      const int h = quotient(2 * i, hd, a.hd_magic), d = 2 * i - h * hd;
      const float* from = sm + h * kPitch;
      float mx = -INFINITY;
#pragma unroll 8
      for (int w = 0; w < used; ++w) mx = fmaxf(mx, from[w * 8 * kPitch + PANELS * 64]);
      float ls = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 4
      for (int w = 0; w < used; ++w) {
        const float* x = from + w * 8 * kPitch;
        const float2 ml = *reinterpret_cast<const float2*>(x + PANELS * 64), v = *reinterpret_cast<const float2*>(x + d);
        const float f = exp2f(ml.x - mx);
        ls += ml.y * f;
        o0 += v.x * f;
        o1 += v.y * f;
      }
      const float inv = inverse(ls);
      const uint32_t v = pack2(divide(o0, ls, inv), divide(o1, ls, inv));
      const size_t at = (size_t)b * (qd / 2) + (size_t)((h0 + h) * hd + d) / 2;
      put_word(a.w_att + at, v, epoch);
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

// ---- temperature sampling (ane/train_full.go:318-342): this CTA's vocabulary range [v0, v1) of every row in double, the
// ranges' sums in order, and the CTA whose range holds the target walks it.  CTA c's range is units of 8 tokens
// [c n / grid, (c + 1) n / grid).  sync() = a grid barrier, false when somebody gave up.
template <int NW, class Sync>
__device__ __forceinline__ bool sample_tokens(const DecodeArgs& a, int step, const unsigned long long* best, double* scratch, int* s_tok,
                                              double* s_before, double* s_target, Sync sync) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int v0 = 8 * (int)((long long)(a.V / 8) * blockIdx.x / gridDim.x), v1 = 8 * (int)((long long)(a.V / 8) * (blockIdx.x + 1) / gridDim.x);
  const double inv_temp = (double)(1.0f / a.temperature);
#pragma unroll 1
  for (int b = warp; b < a.B; b += NW) {
    const double mx = (double)best_value(__ldcg(best + b));
    double s = 0.0;
#pragma unroll 1
    for (int v = v0 + lane; v < v1; v += 32) s += exp(((double)__ldcg(a.logits + (size_t)b * a.V + v) - mx) * inv_temp);
    s = warp_sum_d(s);
    if (lane == 0) __stcg(a.psum + (size_t)blockIdx.x * a.B + b, s);
  }
  if (!sync()) return false;
  double* s_sums = scratch;  // [gridDim.x][B]
#pragma unroll 1
  for (int i = threadIdx.x; i < (int)gridDim.x * a.B; i += NW * 32) s_sums[i] = __ldcg(a.psum + i);
  cta_sync<NW>();
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
  cta_sync<NW>();
#pragma unroll 1
  for (int b = warp; b < a.B; b += NW) {
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
  return sync();
}

enum Kind { kQkv = 0, kWo = 1, kW13 = 2, kW2 = 3, kHead = 4 };

__device__ __forceinline__ const float* norm_gains(const DecodeArgs& a, int kind, int layer) {
  if (kind == kWo || kind == kW2) return nullptr;
  return a.p + (kind == kHead ? a.off_rms_final : (kind == kQkv ? a.off_rms_att : a.off_rms_ffn) + (size_t)layer * a.rms_stride);
}

}  // namespace
}  // namespace ane
