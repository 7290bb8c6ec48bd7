// KV-cached generation for 9 to 32 sequences, and for models too wide for decode.cu (llama-style architecture, bf16 engines):
// all steps after the prefill in one persistent cooperative kernel, with every contraction split over a cluster of four
// CTAs.  32 sequences of the 110M model with 4 KV heads at 512 to 768 positions: 437 -> 398 us a step (the figures below are
// SM cycles of one layer there).
//
// What bounds a phase at these batch sizes is not the weights (95 KB per SM and layer at dim 768) but latency, and the
// activations: an SM that computes whole rows of W x needs all of x -- 98 KB of fp32 at 32 x 768 before a norm, 131 KB for W2 --
// and takes them from L2 at about 30 bytes a cycle, every SM the same ones (6400 to 8500 cycles for a norm).  With the
// contraction split four ways an SM reads a quarter (its columns of all rows), normalises only that, and keeps it in
// registers for all of the cluster's weight rows (3500 cycles).  The price is an exchange of partial sums through
// distributed shared memory, 1 KB per 8 weight rows and CTA, and of the rows' sums of squares.  CTA r of a cluster
// finishes the r-th quarter of the sequences.
//   * Between clusters results travel as flagged words, as in decode.cu: a grid barrier took 3400 to 5700 cycles, five in
//     a layer, the doubled traffic of a quarter takes less.
//   * Inside a cluster they travel by asynchronous stores that count their bytes on a barrier beside the data.
//   * Few warps with many registers: sixteen warps kept spilling what lives across the phases, and with all shared memory
//     taken spilled registers come back from L2 (mma sections of 4500 cycles instead of 1000).
//   * The copies of weights and the prefetches have a warp of their own; one of the computing warps was 1000 cycles late
//     with them in every phase.
//
// Products: mma.sync m16n8k16 -- the sequences are the A rows, 8 weight rows (a "unit") the B columns; a cluster owns a
// contiguous range of every product's units.  Inside a CTA a warp takes one unit of a group and one part of the CTA's
// chunks of 32 columns.  The order of k inside a chunk is free as long as both operands agree, so every lane reads 16
// contiguous bytes of a weight row (k = 8 (lane % 4) ..) and uses them as the fragments of two MMAs: no ldmatrix.
// Weights never change: they stream into a ring of shared-memory slots, as far ahead as the ring reaches, across phases and
// steps, in tensor copies of 8 rows (a quarter of a row is 384 bytes at dim 768; untiled copies of that size arrived at 2.4
// bytes a cycle).
#include <algorithm>

#include "decode_common.cuh"
#include "gemm.h"

namespace ane {
namespace {

constexpr int kWarps = 8, kThreads = kWarps * 32;  // warps that compute; few, with many registers: the latency of a phase counts
constexpr int kLaunch = kThreads + 128;                // and a warpgroup that copies
constexpr int kCluster = 4;
constexpr int kMaxSlots = 8, kMaxUnits = 8;  // slots of the ring; units of a group
constexpr int kKeep = 6;                      // chunks whose A fragments a warp keeps in registers

// One product's share of this CTA (in shared memory): columns [k0, k0 + kn) of the cluster's `nu` units.
struct Slice {
  int K, k0, kn, nc;    // nc chunks of 32 columns
  int box, unit_bytes;  // chunks in a row of a copied box of 8 weight rows; a unit's boxes lie one behind another
  int u0, nu, kind;
  int group, parts_log;  // units per group; warps that share a unit's chunks
  int part_chunks;       // chunks of a warp
  int box_magic;         // q / box = (q * box_magic) >> 16
  // first weight row of the cluster's unit i.  W1 and W3 lie in blocks of 32 rows; units 2j and 2j + 1 are matching rows
  __device__ __forceinline__ int row0(int i) const {
    if (kind != kW13) return (u0 + i) * 8;
    const int pair = (u0 + i) >> 1;
    return (pair >> 2) * 64 + (pair & 3) * 8 + (i & 1) * 32;
  }
};

// Columns of rank r: a quarter of the chunks each, rounded up.
__host__ __device__ inline int chunks_per_cta(int K) { return ((K + 31) / 32 + kCluster - 1) / kCluster; }
// A unit comes in boxes of 8 rows by at most 256 columns, as many chunks each.
__host__ __device__ inline int boxes(int K) { return (chunks_per_cta(K) + 7) / 8; }
__host__ __device__ inline int box_chunks(int K) { return (chunks_per_cta(K) + boxes(K) - 1) / boxes(K); }
__host__ __device__ inline int unit_bytes(int K) { return boxes(K) * box_chunks(K) * 512; }
__device__ __forceinline__ void make_slice(Slice& d, int kind, int K, int units, int group, int rank) {
  const int q = (int)blockIdx.x / kCluster, n = (int)gridDim.x / kCluster, step = kind == kW13 ? 2 : 1, items = units / step;
  const int chunks = (K + 31) / 32, per = chunks_per_cta(K), c0 = min(rank * per, chunks);
  d.K = K;
  d.kind = kind;
  d.k0 = c0 * 32;
  d.nc = min(per, chunks - c0);
  d.kn = max(0, min(d.nc * 32, K - d.k0));
  d.box = box_chunks(K);
  d.unit_bytes = unit_bytes(K);
  d.u0 = step * (int)((long long)items * q / n);
  d.nu = step * (int)((long long)items * (q + 1) / n) - d.u0;
  d.group = group;
  d.parts_log = 0;
  while ((2 << d.parts_log) * min(group, max(d.nu, 1)) <= kWarps && (2 << d.parts_log) <= per) ++d.parts_log;
  d.part_chunks = (per + (1 << d.parts_log) - 1) >> d.parts_log;
  d.box_magic = 65536 / d.box + 1;
}

struct WeightMaps {
  CUtensorMap m[5];       // by product: [layer][row][column], boxes of 8 rows
  CUtensorMap keys, values;  // the caches: [layer][sequence, position][column], boxes of 256 positions of one head
};
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

// One more warp than those that compute streams the weights of the whole generation, in the order they are used, in groups
// of units of one product, each group in one slot of the ring; the norm's gains travel with a product's first group, at
// the slot's end.  full / free = barriers of the slots; a slot is free when every computing warp has arrived there.  The
// lanes issue a unit each.
__device__ __forceinline__ void feed_weights(const DecodeArgs& a, const WeightMaps& maps, const Slice* slices, uint32_t full, uint32_t free, uint32_t ring) {
  const int lane = threadIdx.x & 31;
  int at = 0, issued = 0;
  uint32_t parity = 1;  // of the slot's barriers: the first round waits for nothing
  bool go = true;
#pragma unroll 1
  for (int step = 1; step < a.n_new && go; ++step) {
#pragma unroll 1
    for (int idx = 0; idx <= 4 * a.L && go; ++idx) {
      const int layer = idx >> 2, kind = layer == a.L ? kHead : idx & 3;
      const Slice& p = slices[kind];
      if (p.kn == 0) continue;
#pragma unroll 1
      for (int g0 = 0; g0 < p.nu; g0 += p.group) {
        const int n = min(p.group, p.nu - g0);
        const uint32_t b = full + 8u * at, to = ring + (uint32_t)(at * a.slot_bytes), gain_bytes = (uint32_t)p.kn * 4u;
        const float* gains = g0 == 0 ? norm_gains(a, kind, layer) : nullptr;
        if (!mbar_wait(free + 8u * at, parity, a.status, DEV_GRID_TIMEOUT)) {
          go = false;
          break;
        }
        __syncwarp();
        if (lane == 0) {
          mbar_expect_tx(b, (uint32_t)(n * p.unit_bytes) + (gains ? gain_bytes : 0u));
          if (gains) bulk_copy(to + (uint32_t)a.slot_bytes - gain_bytes, gains + p.k0, gain_bytes, b);
        }
        __syncwarp();
        if (lane < n)  // what lies past the row's end arrives as zeros
          for (int k = 0, i = 0; k < p.unit_bytes; k += p.box * 512, ++i)
            tma_load_3d(to + (uint32_t)(lane * p.unit_bytes + k), &maps.m[kind], b, p.k0 + i * p.box * 32, p.row0(g0 + lane), kind == kHead ? 0 : layer);
        __syncwarp();
        ++issued;
        if (++at == a.slots) at = 0, parity ^= 1u;
      }
    }
  }
  // no copy may still be on its way into this CTA's shared memory when it ends (a wait for a phase that has passed is none)
  if (!go)
    for (int i = max(0, issued - a.slots); i < issued; ++i) mbar_wait(full + 8u * (i % a.slots), (uint32_t)(i / a.slots) & 1u, nullptr, 0);
}

// Stores into the shared memory of a CTA of the cluster that count their bytes on a barrier beside the data: the reader
// waits for the bytes, and nobody needs a fence (barrier.cluster.arrive.release took 1000 cycles behind plain stores).
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, float2 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(v.x), "f"(v.y), "r"(bar) : "memory");
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, float v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v), "r"(bar) : "memory");
}

// Waits for one pair of words a lane: cheap polls while the producers are at work, before a warp asks for everything.
__device__ __forceinline__ void await_words(const uint2* p, bool take, uint32_t epoch, const Wait& wait) {
  long long t0 = 0;
#pragma unroll 1
  for (unsigned n = 0;; ++n)
    if (__all_sync(0xffffffffu, words_are(get_words_if(p, take, epoch), epoch)) || wait.expired(n, t0)) return;
}

// stage[chunk][8-row group][lane]: byte offset of element k (from the CTA's first column) of row r.  Rows past the batch
// stay zero from the start.
template <int R8>
__device__ __forceinline__ int frag_at(int r, int k) {
  return ((((k >> 5) * R8 + (r >> 3)) * 32 + (r & 7) * 4 + ((k & 31) >> 3)) << 4) + (k & 7) * 2;
}

// R8: 8-row groups of the batch; PANELS: 64 dims of a head each
template <int R8, int PANELS>
__global__ void __launch_bounds__(kLaunch, 1) decode_batch_kernel(const __grid_constant__ DecodeArgs a, const __grid_constant__ WeightMaps maps) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_tok[32], s_abort;
  __shared__ float s_leave;  // 1: give up
  __shared__ float s_sq[kCluster][32], s_cos[64], s_sin[64];
  __shared__ __align__(8) uint64_t s_full[kMaxSlots], s_free[kMaxSlots], s_sums[2], s_squares, s_go;
  __shared__ unsigned long long s_best[32];
  __shared__ double s_before[32], s_target[32];
  __shared__ Slice s_slice[5];
  constexpr int BP = 8 * R8, T = R8 / 2;     // rows of the batch, their 16-row tiles
  constexpr int Own = BP / kCluster;         // rows that this CTA finishes
  constexpr int EL = Own * 4;                // their column pairs in one unit
  constexpr int kPart = EL * kWarps * kCluster;  // float2 in one buffer of partial sums: [rank][part][unit][row][column pair]
  uint8_t* stage = smem;
  uint8_t* ring = smem + a.stage_bytes;
  float2* part = reinterpret_cast<float2*>(ring + a.slots * a.slot_bytes);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int rank = (int)cluster_ctarank();
  const int D = a.D, QD = a.H * a.hd, KVD = a.KV * a.hd;
  const bool sampling = a.temperature > 1e-6f;
  if (threadIdx.x == 0) {
    s_abort = 0;
    s_leave = 0.f;
    make_slice(s_slice[kQkv], kQkv, D, (QD + 2 * KVD) / 8, a.units, rank);
    make_slice(s_slice[kWo], kWo, QD, D / 8, a.units, rank);
    make_slice(s_slice[kW13], kW13, D, 2 * a.Hd / 8, a.units, rank);
    make_slice(s_slice[kW2], kW2, a.Hd, D / 8, a.units_w2, rank);
    make_slice(s_slice[kHead], kHead, D, a.V / 8, a.units, rank);
  }
  for (int i = threadIdx.x * 16; i < a.stage_bytes; i += kLaunch * 16) *reinterpret_cast<uint4*>(stage + i) = make_uint4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    for (int i = 0; i < a.slots; ++i) {
      mbar_init(smem_u32(s_full) + 8u * i, 1);
      mbar_init(smem_u32(s_free) + 8u * i, kWarps);
    }
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(s_sums) + 8u * i, 1);
    mbar_init(smem_u32(&s_squares), 1);
    mbar_init(smem_u32(&s_go), 1);
    fence_mbar_init();
  }
  cluster_sync_all();  // every CTA of the cluster runs before anybody writes into its shared memory
  // 384 threads start with 168 registers each; two warpgroups compute with 224, the third keeps 56 and copies.
  if (warp >= kWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == kWarps) feed_weights(a, maps, s_slice, smem_u32(s_full), smem_u32(s_free), smem_u32(ring));
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    [&] {
      const Wait wait{a.status, &s_abort};
      int slot = 0;        // the next group's slot, and the parity of its barrier
      uint32_t parity = 0;
      auto wait_for = [&](uint32_t bar, uint32_t phase) {
        if (s_abort == 0 && !mbar_wait(bar, phase, a.status, DEV_GRID_TIMEOUT)) s_abort = 1;
        __syncwarp();
      };
      auto group_ready = [&] { wait_for(smem_u32(&s_full[slot]), parity); };
      // Grid barrier: every CTA arrives, rank 0 of each cluster waits for the count and tells the others.  The four CTAs of a
      // cluster give up together, so that nobody writes into the shared memory of one that has left.
      unsigned target = 0;
      uint32_t go_parity = 0;
      const uint32_t leave_at = smem_u32(&s_leave);
      auto grid_arrive = [&] {
        target += gridDim.x;
        cta_sync<kWarps>();
        if (threadIdx.x == 0) asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        __syncwarp();
      };
      auto grid_wait = [&]() -> bool {
        if (threadIdx.x == 0) mbar_expect_tx(smem_u32(&s_go), sizeof(float));
        if (rank == 0 && threadIdx.x == 0) {
          unsigned seen;
          long long t0 = 0;
          float left = 0.f;
#pragma unroll 1
          for (unsigned n = 0;; ++n) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
            if ((int)(seen - target) >= 0) break;
            if (wait.expired(n, t0)) {
              left = 1.f;
              break;
            }
          }
          for (uint32_t i = 0; i < kCluster; ++i) send(map_to_cta(leave_at, i), map_to_cta(smem_u32(&s_go), i), left);
        }
        __syncwarp();
        if (!mbar_wait(smem_u32(&s_go), go_parity, a.status, DEV_GRID_TIMEOUT)) s_leave = 1.f;
        go_parity ^= 1u;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        cta_sync<kWarps>();
        return *reinterpret_cast<volatile float*>(&s_leave) == 0.f;
      };
      // The cached keys and values that this CTA will attend to, from DRAM into L2 ahead of the attention, whose own loads
      // are a chain of a few.  (One request per 256 positions: a prefetch instruction per row kept the load unit busy for
      // 2000 cycles.)
      auto prefetch_kv = [&](int l, int pos) {
        if (warp == 1) {
          int group = a.group, hd = a.hd;
          asm volatile("" : "+r"(group), "+r"(hd));  // see attention_phase()
          const int hgroups = a.items, box = min(256, a.S);
          for (int item = blockIdx.x; item < a.B * hgroups; item += gridDim.x) {
            const int b = quotient(item, hgroups, a.items_magic), kvh = quotient((item - b * hgroups) * group, a.rep, a.rep_magic);
            for (int j = lane * box; j < pos; j += 32 * box) {
              asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(&maps.keys)), "r"(kvh * hd),
                           "r"(b * a.S + j), "r"(l) : "memory");
              asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(&maps.values)),
                           "r"(kvh * hd), "r"(b * a.S + j), "r"(l) : "memory");
            }
          }
        }
        __syncwarp();
      };
      // where this lane's partial sums go: rows 0-7 and 8-15 of each tile belong to different CTAs
      uint32_t to[T][2], sums[T][2];
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = t * 16 + h * 8 + g;
          to[t][h] = map_to_cta(smem_u32(part), (uint32_t)(row / Own)) + (uint32_t)((row % Own) * 4 + c) * 8u;
          sums[t][h] = map_to_cta(smem_u32(s_sums), (uint32_t)(row / Own));
        }
      const int er = (threadIdx.x / 4) % Own, brow = rank * Own + er;  // the epilogues' row
      const bool live = brow < a.B;
      int buf = 0;  // buffer of partial sums
      uint32_t sums_parity = 0, squares_parity = 0;  // sums_parity: bit per buffer

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
        cta_sync<kWarps>();
        float bv = -INFINITY;
        int bi = -1;
        // the phases of the step in order: q|k|v, attention, Wo, W1|W3 and W2 of every layer, and the classifier.  (One copy of
        // the code for all products: it stays in the instruction cache.)
#pragma unroll 1
        for (int l = 0, phase = 0;;) {
          const int kind = l == a.L ? kHead : phase == 0 ? kQkv : phase - 1;
          const uint32_t epoch = (uint32_t)(step * a.L + l + 1);
          if (phase == 1) {
            const size_t cl = (size_t)l * a.kv_layer;
            float* sm = reinterpret_cast<float*>(part + 2 * kPart);  // (the others of the cluster may be sending sums)
            attention_phase<PANELS, kWarps, PANELS == 1 ? 2 : 1>(a, a.kcache + cl, a.vcache + cl, pos, sm, epoch, wait);
          } else {
            const Slice& p = s_slice[kind];
            auto residual = [&](int col) {  // x before this product: the embedding, or words that this cluster has staged
              if (kind == kWo && l == 0) return __ldg(reinterpret_cast<const float2*>(a.p + a.off_embed_f32 + (size_t)s_tok[brow] * D + col));
              const uint4 o = get_words((kind == kWo ? a.w_x0 : a.w_x1) + (size_t)brow * D + col);
              return make_float2(__uint_as_float(o.x), __uint_as_float(o.z));
            };
            float2 old = make_float2(0.f, 0.f);
            if (kind == kWo || kind == kW2) {
              // bf16 rows, this CTA's columns, into fragment order
              constexpr int N = BP / kWarps;
              const uint2* words = (kind == kWo ? a.w_att : a.w_gate) + p.k0 / 2;
#pragma unroll 1
              for (int k0 = lane * 8; p.nu > 0 && k0 - lane * 8 < p.kn; k0 += 512) {
                await_words(words + ((size_t)warp * p.K + k0) / 2, warp < a.B && k0 < p.kn, epoch, wait);
                uint4 w[N][2][2];
                long long t0 = 0;
#pragma unroll 1
                for (unsigned n = 0;; ++n) {
                  bool ok = true;
#pragma unroll
                  for (int i = 0; i < N; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                      const int r = warp + i * kWarps, k = k0 + h * 256;
                      const uint2* at = words + ((size_t)r * p.K + k) / 2;
                      w[i][h][0] = get_words_if(at, r < a.B && k < p.kn, epoch);
                      w[i][h][1] = get_words_if(at + 2, r < a.B && k < p.kn, epoch);
                    }
#pragma unroll
                  for (int i = 0; i < N; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) ok = ok && words_are(w[i][h][0], epoch) && words_are(w[i][h][1], epoch);
                  if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
                }
#pragma unroll
                for (int i = 0; i < N; ++i)
#pragma unroll
                  for (int h = 0; h < 2; ++h) {
                    const int r = warp + i * kWarps, k = k0 + h * 256;
                    if (r < a.B && k < p.kn) *reinterpret_cast<uint4*>(stage + frag_at<R8>(r, k)) = make_uint4(w[i][h][0].x, w[i][h][0].z, w[i][h][1].x, w[i][h][1].z);
                  }
              }
              if (live && (int)threadIdx.x < min(p.group, p.nu) * EL) old = residual(p.row0(threadIdx.x / EL) + 2 * (threadIdx.x & 3));  // of this thread's first pair
            } else {
              // Normalised rows, bf16(x * rms^-1 * gain), rounded like the training forward's.  A thread's part of a row stays
              // in registers between the sum of squares and the conversion for dim <= 768; wider rows are read twice.
              constexpr int V = 6, Per = kThreads / BP, Seg = Per * 4 * V;
              const int r = threadIdx.x / Per, sub = threadIdx.x % Per, nseg = max(1, (p.kn + Seg - 1) / Seg);
              const bool has = r < a.B;
              const bool embed = kind == kQkv && l == 0;
              const uint32_t want = kind == kW13 ? epoch : epoch - 1;
              const float* px = a.p + a.off_embed_f32 + (size_t)(embed && has ? s_tok[r] : 0) * D + p.k0;
              const uint2* pw = (kind == kW13 ? a.w_x1 : a.w_x0) + (size_t)(has ? r : 0) * D + p.k0;
              const float* gains = reinterpret_cast<const float*>(ring + (slot + 1) * a.slot_bytes - p.kn * 4);
              float sq = 0.f, rms = 0.f;
#pragma unroll 1
              for (int it = 0; it < (nseg == 1 ? 1 : 2 * nseg); ++it) {
                const int k = (it < nseg ? it : it - nseg) * Seg + sub * 4;
                float4 x[V];
#pragma unroll
                for (int i = 0; i < V; ++i) x[i] = ldf_l2_if(px + k + i * Per * 4, embed && has && k + i * Per * 4 < p.kn);
                if (!embed) {
                  await_words(pw + k, has && k < p.kn, want, wait);
                  long long t0 = 0;
#pragma unroll 1
                  for (unsigned n = 0;; ++n) {
                    bool ok = true;
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                      const bool take = has && k + i * Per * 4 < p.kn;
                      const uint4 u = get_words_if(pw + k + i * Per * 4, take, want), v = get_words_if(pw + k + i * Per * 4 + 2, take, want);
                      ok = ok && words_are(u, want) && words_are(v, want);
                      x[i] = make_float4(__uint_as_float(u.x), __uint_as_float(u.z), __uint_as_float(v.x), __uint_as_float(v.z));
                    }
                    if (__all_sync(0xffffffffu, ok) || wait.expired(n, t0)) break;
                  }
                }
                if (it < nseg) {
#pragma unroll
                  for (int i = 0; i < V; ++i) sq += (x[i].x * x[i].x + x[i].y * x[i].y) + (x[i].z * x[i].z + x[i].w * x[i].w);
                }
                if (it == nseg - 1) {
#pragma unroll
                  for (int o = Per / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
                  if (threadIdx.x == 0) mbar_expect_tx(smem_u32(&s_squares), sizeof(float) * kCluster * BP);
                  if (sub < kCluster) send(map_to_cta(smem_u32(&s_sq[rank][r]), (uint32_t)sub), map_to_cta(smem_u32(&s_squares), (uint32_t)sub), sq);
                  __syncwarp();
                  if (p.nu > 0 && p.kn > 0) group_ready();
                  wait_for(smem_u32(&s_squares), squares_parity);
                  squares_parity ^= 1u;
                  sq = (s_sq[0][r] + s_sq[1][r]) + (s_sq[2][r] + s_sq[3][r]);
                  rms = inverse_sqrt(fmaf(sq, a.inv_dim, 1e-5f));
                }
                if ((it >= nseg || nseg == 1) && p.nu > 0) {
#pragma unroll
                  for (int i = 0; i < V; ++i) {
                    if (!has || k + i * Per * 4 >= p.kn) continue;
                    const float4 w = *reinterpret_cast<const float4*>(gains + k + i * Per * 4);
                    *reinterpret_cast<uint2*>(stage + frag_at<R8>(r, k + i * Per * 4)) =
                        make_uint2(pack2(x[i].x * rms * w.x, x[i].y * rms * w.y), pack2(x[i].z * rms * w.z, x[i].w * rms * w.w));
                  }
                }
              }
            }
            cta_sync<kWarps>();
            // this warp's unit of every group and its chunks
            const int unit = warp >> p.parts_log, kp = warp & ((1 << p.parts_log) - 1), parts = 1 << p.parts_log;
            const int c0 = kp * p.part_chunks, nc = max(0, min(p.part_chunks, p.nc - c0));
            const uint4* st = reinterpret_cast<const uint4*>(stage) + (size_t)c0 * R8 * 32 + lane;
            const int last = max(nc - 1, 0);  // loads go by clamped chunks: no branches between them
            uint4 f[kKeep][R8];
#pragma unroll
            for (int i = 0; i < kKeep; ++i)
#pragma unroll
              for (int r = 0; r < R8; ++r) f[i][r] = st[(min(i, last) * R8 + r) * 32];
            const int box = p.box, box_magic = p.box_magic;
            auto finish = [&](int g0) {
              const int n = min(p.group, p.nu - g0);
              wait_for(smem_u32(&s_sums[buf ^ 1]), (sums_parity >> (buf ^ 1)) & 1u);  // all partial sums have arrived
              sums_parity ^= 1u << (buf ^ 1);
              const float2* from = part + (buf ^ 1) * kPart + (threadIdx.x % EL);
              auto sum = [&](int u) {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll 4
                for (int i = 0; i < kCluster * parts; ++i) {
                  const float2 v = from[(i * n + u) * EL];
                  s.x += v.x;
                  s.y += v.y;
                }
                return s;
              };
              const int e = threadIdx.x / EL;  // unit, or pair of units for W1|W3
              static_assert(kMaxUnits * EL <= kThreads);
              if (!live) {
              } else if (kind == kW13) {
                if (e < n / 2) {
                  const float2 h1 = sum(2 * e), h3 = sum(2 * e + 1);
                  const int col = ((p.u0 + g0) / 2 + e) * 8 + 2 * (threadIdx.x & 3);
                  put_word(a.w_gate + ((size_t)brow * a.Hd + col) / 2, pack2(h1.x * h3.x * sigmoid(h1.x), h1.y * h3.y * sigmoid(h1.y)), epoch);
                }
              } else if (e < n) {
                float2 s = sum(e);
                const int col = p.row0(g0 + e) + 2 * (threadIdx.x & 3);
                if (kind == kQkv) {
                  if (col < QD + KVD) {
                    const int r = (col - (int)__umulhi((unsigned)col, a.hd_magic) * a.hd) >> 1;
                    s = make_float2(s.x * s_cos[r] - s.y * s_sin[r], s.y * s_cos[r] + s.x * s_sin[r]);
                  }
                  const uint32_t v = pack2(s.x, s.y);
                  put_word(a.w_qkv + ((size_t)brow * (QD + 2 * KVD) + col) / 2, v, epoch);
                  if (col >= QD) {
                    bf16* cache = (col < QD + KVD ? a.kcache + (col - QD) : a.vcache + (col - QD - KVD)) + (size_t)l * a.kv_layer;
                    __stcg(reinterpret_cast<unsigned*>(cache + ((size_t)brow * a.S + pos) * KVD), v);
                  }
                } else if (kind == kHead) {
                  if (s.x > bv) { bv = s.x; bi = col; }
                  if (s.y > bv) { bv = s.y; bi = col + 1; }
                  if (sampling) __stcg(reinterpret_cast<float2*>(a.logits + (size_t)brow * a.V + col), s);
                } else {  // x += product; every element is updated by one thread
                  if (g0 > 0) old = residual(col);
                  uint2* to = (kind == kWo ? a.w_x1 : a.w_x0) + (size_t)brow * D + col;
                  put_word(to, __float_as_uint(s.x + old.x), epoch);
                  put_word(to + 1, __float_as_uint(s.y + old.y), epoch);
                }
              }
              __syncwarp();
            };
#pragma unroll 1
            for (int g0 = 0;; g0 += p.group) {  // the products of a group run while the sums of the one before travel
              const bool more = g0 < p.nu;
              float acc[T][4] = {};
              if (more && p.kn > 0) group_ready();
              __syncwarp();
              if (more && unit < min(p.group, p.nu - g0)) {
                const uint8_t* wp = ring + slot * a.slot_bytes + unit * p.unit_bytes + g * box * 64 + c * 16;
#pragma unroll 1
                for (int blk = 0; blk < nc; blk += kKeep) {
                  if (nc > kKeep && (blk > 0 || g0 > 0)) {  // that many chunks or fewer: the same fragments for every group
#pragma unroll
                    for (int i = 0; i < kKeep; ++i)
#pragma unroll
                      for (int r = 0; r < R8; ++r) f[i][r] = st[(min(blk + i, last) * R8 + r) * 32];
                  }
                  uint4 b[kKeep];
#pragma unroll
                  for (int i = 0; i < kKeep; ++i) {
                    const int q = c0 + min(blk + i, last), at_box = (q * box_magic) >> 16;  // q / box
                    b[i] = *reinterpret_cast<const uint4*>(wp + at_box * box * 448 + q * 64);
                  }
#pragma unroll
                  for (int i = 0; i < kKeep; ++i) {
                    if (blk + i < nc) {
#pragma unroll
                      for (int t = 0; t < T; ++t) {
                        const uint4 lo = f[i][2 * t], hi = f[i][2 * t + 1];
                        mma16816(acc[t], lo.x, hi.x, lo.y, hi.y, b[i].x, b[i].y);
                        mma16816(acc[t], lo.z, hi.z, lo.w, hi.w, b[i].z, b[i].w);
                      }
                    }
                  }
                }
              }
              if (more && p.kn > 0) {
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_free[slot]));
                if (++slot == a.slots) slot = 0, parity ^= 1u;
              }
              if (g0 > 0) finish(g0 - p.group);
              if (!more) break;
              // All warps have left the sums of the group before: what this CTA sends now tells the others so.
              cta_sync<kWarps>();
              const int n = min(p.group, p.nu - g0);
              if (threadIdx.x == 0) mbar_expect_tx(smem_u32(&s_sums[buf]), (uint32_t)(8 * EL * kCluster * n) << p.parts_log);
              if (unit < n) {
                const uint32_t at = (uint32_t)(buf * kPart + (((rank << p.parts_log) + kp) * n + unit) * EL) * 8u;
#pragma unroll
                for (int t = 0; t < T; ++t) {
                  send(to[t][0] + at, sums[t][0] + 8u * buf, make_float2(acc[t][0], acc[t][1]));
                  send(to[t][1] + at, sums[t][1] + 8u * buf, make_float2(acc[t][2], acc[t][3]));
                }
              }
              __syncwarp();
              buf ^= 1;
            }
          }
          if (l == a.L) break;
          if (phase == 4 && l + 1 < a.L) prefetch_kv(l + 1, pos);
          if (++phase == 5) {
            phase = 0;
            ++l;
          }
        }
        // ---- the best logit of every row
        if (bi >= 0) atomicMax(&s_best[brow], pack_best(bv, bi));
        cta_sync<kWarps>();
        if ((int)threadIdx.x < a.B && s_best[threadIdx.x] != 0) atomicMax(best + threadIdx.x, s_best[threadIdx.x]);
        grid_arrive();
        if (step + 1 < a.n_new) prefetch_kv(0, pos);
        auto sync = [&] {
          grid_arrive();
          return grid_wait();
        };
        if (!grid_wait() || (sampling && !sample_tokens<kWarps>(a, step, best, reinterpret_cast<double*>(part), s_tok, s_before, s_target, sync))) {
          return;
        }
      }
      if (!sampling && a.n_new > 1 && blockIdx.x == 0 && (int)threadIdx.x < a.B) {
        const unsigned long long k = __ldcg(a.best + ((a.n_new - 1) % 3) * a.B + threadIdx.x);
        a.out[(size_t)threadIdx.x * a.n_new + a.n_new - 1] = (uint16_t)(k == 0 ? 0 : 0xffffffffu - (uint32_t)k);
      }
    }();
  }
  cluster_sync_all();  // (nothing of the exchange is on its way into a CTA that has left)
}

struct Plan {
  int r8, stage_bytes, slot_bytes, slots, units, units_w2;
  size_t smem;
};
constexpr size_t kSmemLimit = 222 * 1024;  // beside the static arrays

Plan make_plan(int D, int Hd, int hd, int ctas, int batch) {
  Plan p;
  p.r8 = batch <= 16 ? 2 : 4;
  p.stage_bytes = std::max(chunks_per_cta(D), chunks_per_cta(Hd)) * p.r8 * 512;
  // partial sums, two buffers, and the attention's merge; the sampler uses the same memory
  const size_t sums = 2 * sizeof(float2) * (size_t)(8 * p.r8 * kWarps * 4), merge = sizeof(float) * (size_t)(kWarps * 8 * (2 + (hd <= 64 ? 64 : 128)));
  const size_t tail = std::max(sums + merge, sizeof(double) * (size_t)ctas * batch);
  for (p.units = kMaxUnits;; p.units /= 2) {  // fewer units in a group where three slots would not fit
    p.slot_bytes = std::max(p.units * unit_bytes(D) + chunks_per_cta(D) * 128, unit_bytes(Hd));
    p.units_w2 = std::min(kMaxUnits, p.slot_bytes / unit_bytes(Hd));
    const size_t room = kSmemLimit > p.stage_bytes + tail ? kSmemLimit - p.stage_bytes - tail : 0;
    p.slots = (int)std::min<size_t>(kMaxSlots, room / p.slot_bytes);
    if (p.slots >= 3 || p.units == 2) break;
  }
  p.smem = p.stage_bytes + (size_t)p.slots * p.slot_bytes + tail;
  return p;
}

}  // namespace

bool decode_batch_supported(int D, int Hd, int hd, int batch, int sms) { return make_plan(D, Hd, hd, sms, batch).slots >= 2; }

int decode_batch_steps(DecodeArgs a, int sms, cudaStream_t s) {
  const Plan p = make_plan(a.D, a.Hd, a.hd, sms, a.B);
  WeightMaps maps;
  auto map = [&](int kind, size_t off, int K, int rows, int layers) {
    return make_tmap_weights(&maps.m[kind], a.w + off, (uint64_t)K, (uint64_t)rows, (uint64_t)layers, a.layer_stride, (uint32_t)box_chunks(K) * 32, 8);
  };
  if (!map(kQkv, a.off_qkv, a.D, (a.H + 2 * a.KV) * a.hd, a.L) || !map(kWo, a.off_wo, a.H * a.hd, a.D, a.L) ||
      !map(kW13, a.off_w13, a.D, 2 * a.Hd, a.L) || !map(kW2, a.off_w2, a.Hd, a.D, a.L) || !map(kHead, a.off_embed, a.D, a.V, 1) ||
      !make_tmap_weights(&maps.keys, a.kcache, (uint64_t)a.KV * a.hd, (uint64_t)a.B * a.S, (uint64_t)a.L, a.kv_layer, (uint32_t)a.hd, (uint32_t)std::min(256, a.S)) ||
      !make_tmap_weights(&maps.values, a.vcache, (uint64_t)a.KV * a.hd, (uint64_t)a.B * a.S, (uint64_t)a.L, a.kv_layer, (uint32_t)a.hd, (uint32_t)std::min(256, a.S)))
    return -2;
  a.stage_bytes = p.stage_bytes;
  a.slot_bytes = p.slot_bytes;
  a.slots = p.slots;
  a.units = p.units;
  a.units_w2 = p.units_w2;
  auto kern = a.hd <= 64 ? (p.r8 == 2 ? decode_batch_kernel<2, 1> : decode_batch_kernel<4, 1>) : (p.r8 == 2 ? decode_batch_kernel<2, 2> : decode_batch_kernel<4, 2>);
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem) != cudaSuccess) return -3;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;  // all CTAs are resident together, so the waits on one another complete
  attr[1].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  if (sms < kCluster) return -4;
  cfg.gridDim = dim3((unsigned)(sms / kCluster * kCluster));
  cfg.blockDim = dim3(kLaunch);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;  // a cluster's CTAs share a part of the chip, so fewer than sms / 4 may fit
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters <= 0) return -3;
  // every cluster owns units of q|k|v and of W1|W3: see put_word()
  clusters = std::min({clusters, sms / kCluster, (a.H + 2 * a.KV) * a.hd / 8, a.Hd / 8});
  cfg.gridDim = dim3((unsigned)(clusters * kCluster));
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, a, maps) == cudaSuccess ? 0 : -4;
}

}  // namespace ane
