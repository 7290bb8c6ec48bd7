// GEMM launchers: tcgen05 bf16 path (gemm_tc.cuh), fp32 products on the tensor cores (gemm_f32_tc.cuh) and on the FMA units.
#include "gemm.h"

#include <cuda.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "gemm_f32_tc.cuh"
#include "gemm_tc.cuh"

namespace ane {

static thread_local std::string g_gemm_err;
const char* gemm_last_error() { return g_gemm_err.c_str(); }

bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("ANE_B200_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

int gemm_num_sms() {
  static int sms[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (sms[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    // ANE_B200_GEMM_SMS caps the persistent grids (e.g. to leave SMs to a communication kernel).
    const char* e = getenv("ANE_B200_GEMM_SMS");
    if (e && atoi(e) > 0 && atoi(e) < n) n = atoi(e);
    sms[dev] = n;
  }
  return sms[dev];
}

// ------------------------------------------------------------------------------------------
// Tensor maps
// ------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// 2-D tensor [outer, inner] with row pitch ld (elements); box = [box_outer, box_inner]; 128B swizzle.
static bool make_tmap(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer, bool is_f32 = false) {
  // Encoding takes about a microsecond and a step asks for some 700 maps of buffers that never move: a small direct-mapped
  // cache per thread (no lock; a shared std::map behind a mutex cost several tenths of a microsecond per map).
  struct Key {
    const void* ptr;
    uint64_t inner, outer, ld;
    uint32_t box_inner, box_outer;
    int dev, f32;
    bool operator==(const Key& o) const {
      return ptr == o.ptr && inner == o.inner && outer == o.outer && ld == o.ld && box_inner == o.box_inner && box_outer == o.box_outer &&
             dev == o.dev && f32 == o.f32;
    }
  };
  struct Entry {
    CUtensorMap tm;
    Key key;
  };
  constexpr size_t kEntries = 2048;
  static thread_local std::vector<Entry> cache;
  if (cache.empty()) cache.resize(kEntries);  // zero keys match no call: a null pointer is refused below
  int dev = 0;
  cudaGetDevice(&dev);
  const Key key{ptr, inner, outer, ld, box_inner, box_outer, dev, is_f32 ? 1 : 0};
  uint64_t h = reinterpret_cast<uintptr_t>(ptr) >> 4;
  for (uint64_t v : {inner, outer, ld, (uint64_t)box_inner << 32 | box_outer, (uint64_t)dev << 1 | (uint64_t)key.f32})
    h = (h ^ v) * 0x9E3779B97F4A7C15ull;
  Entry& entry = cache[(h >> 40) % kEntries];
  const uint64_t esz = is_f32 ? 4 : 2;
  if (ptr != nullptr && entry.key == key) {
    *out = entry.tm;
    return true;
  }
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) {
    g_gemm_err = "cuTensorMapEncodeTiled entry point not available";
    return false;
  }
  if (ptr == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (ld * esz) % 16 != 0) {
    g_gemm_err = "TMA operand must be 16-byte aligned with a 16-byte multiple row pitch";
    return false;
  }
  cuuint64_t gdim[2] = {inner, outer};
  cuuint64_t gstride[1] = {ld * esz};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMap tm;
  CUresult r = fn(&tm, is_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed (%d) inner=%llu outer=%llu ld=%llu", (int)r,
             (unsigned long long)inner, (unsigned long long)outer, (unsigned long long)ld);
    g_gemm_err = buf;
    return false;
  }
  entry.tm = tm;
  entry.key = key;
  *out = tm;
  return true;
}

bool make_tmap_2d(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_inner,
                  uint32_t box_outer, bool is_f32) {
  return make_tmap(out, ptr, inner, outer, ld, box_inner, box_outer, is_f32);
}

// [layer][row][column] bf16 matrices, dense rows, `layer_stride` elements apart; boxes of box_rows x box_inner, not swizzled.
bool make_tmap_weights(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t rows, uint64_t layers, uint64_t layer_stride,
                       uint32_t box_inner, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) {
    g_gemm_err = "cuTensorMapEncodeTiled entry point not available";
    return false;
  }
  cuuint64_t gdim[3] = {inner, rows, layers}, gstride[2] = {inner * 2, (layers > 1 ? layer_stride : rows * inner) * 2};
  cuuint32_t box[3] = {box_inner, box_rows, 1}, estr[3] = {1, 1, 1};
  if (fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
    return true;
  g_gemm_err = "cuTensorMapEncodeTiled failed for a weight matrix";
  return false;
}

template <int BN, int MT, bool A_MN, bool B_MN, int EPI>
static int launch_tc(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& td,
                     const EpiParams& epi,
                     const GemmDesc& d, int split_k, int* d_status, cudaStream_t stream) {
  auto kern = gemm_tc_kernel<BN, MT, A_MN, B_MN, EPI>;
  constexpr int threads = 64 + 32 * GemmCfg<BN, MT>::epi_warps(EPI);
  constexpr uint32_t smem_bytes = GemmCfg<BN, MT>::smem_bytes(EPI);
  static_assert(GemmCfg<BN, MT>::fits(EPI), "pipeline does not fit");
  static bool attr_set = false;  // per template instantiation
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
    if (e != cudaSuccess) {
      g_gemm_err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
      return -3;
    }
    attr_set = true;
  }
  constexpr int BM_TILE = GemmCfg<BN, MT>::BM_TILE;
  const int base_tiles = ((d.M + BM_TILE - 1) / BM_TILE) * ((d.N + BN - 1) / BN);
  if constexpr (GemmCfg<BN, MT>::PAIR) {
    // one cluster of two CTAs per tile; as many clusters as the device keeps resident at once
    static int max_pairs = 0;  // per template instantiation
    if (max_pairs == 0) {
      cudaLaunchConfig_t q = {};
      q.gridDim = dim3(2 * 74);
      q.blockDim = dim3(threads);
      q.dynamicSmemBytes = smem_bytes;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      q.attrs = at;
      q.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &q) != cudaSuccess || n <= 0) n = gemm_num_sms() / 2;
      if (n > gemm_num_sms() / 2) n = gemm_num_sms() / 2;
      max_pairs = n;
    }
    const int work = base_tiles * (split_k > 0 ? split_k : 1);
    const int pairs = work < max_pairs ? work : max_pairs;
    cudaError_t e = launch_pdl_cluster(kern, dim3(2 * (pairs < 1 ? 1 : pairs)), dim3(threads), smem_bytes, stream, 2u,
                                       ta, tb, tc, td, epi, d.M, d.N, d.K, split_k > 0 ? split_k : 1, d_status,
                                       (const GemmGroup*)nullptr);
    if (e != cudaSuccess) {
      g_gemm_err = std::string("gemm_tc pair launch: ") + cudaGetErrorString(e);
      return -4;
    }
    return 0;
  }
  int grid;
  if (split_k > 0) {
    const int tiles = base_tiles * split_k;
    grid = tiles < gemm_num_sms() ? tiles : gemm_num_sms();
  } else {  // stream-K: equal shares of the tile x k-block units, at least 8 k-blocks per CTA
    const long long units = (long long)base_tiles * ((d.K + GEMM_BK - 1) / GEMM_BK);
    long long g = units / 8;
    if (g > gemm_num_sms()) g = gemm_num_sms();
    grid = (int)g;
  }
  if (grid < 1) grid = 1;
  cudaError_t e = launch_pdl(kern, dim3(grid), dim3(threads), smem_bytes, stream, ta, tb, tc, td, epi, d.M, d.N,
                             d.K, split_k, d_status, (const GemmGroup*)nullptr);
  if (e != cudaSuccess) {
    g_gemm_err = std::string("gemm_tc launch: ") + cudaGetErrorString(e);
    return -4;
  }
  return 0;
}

template <int BN, int MT, bool A_MN, bool B_MN>
static int dispatch_epi(const CUtensorMap& ta, const CUtensorMap& tb, const GemmDesc& d, int split_k,
                        int* d_status, cudaStream_t stream) {
  EpiParams epi{d.alpha, d.res1, d.s1, d.res2, d.s2, d.ldres, reinterpret_cast<bf16*>(d.aux), d.ldaux,
                d.rope_cos, d.rope_sin, d.rope_seq, d.rope_pos0, d.rope_cols, d.tgt, d.tgt_out, d.tgt_row0,
                d.ce_stats, d.ce_lse2, d.ce_coef, d.ce_rows, d.ce_col0, d.ce_softcap ? 1 : 0, d.part_rows, d.seg_kb};
  if (d.seg_kb > 0) {
    epi.lo_a = d.lda / 2;
    epi.lo_b = d.ldb / 2;
  }
  constexpr int whole = 1;  // schedule of the epilogues that need whole tiles
  constexpr bool NARROW = GemmCfg<BN, MT>::NARROW;
  CUtensorMap tc;
  if constexpr (BN == 32) {
    if (d.out != GEMM_OUT_F32) {
      g_gemm_err = "32-column tiles are built for the fp32 store";
      return -2;
    }
  } else {
  if (d.out == GEMM_OUT_BF16) {
    if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false)) return -2;
    return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_BF16>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
  }
  if (d.out == GEMM_OUT_BF16_TGT) {
    if constexpr (!A_MN && !B_MN && !NARROW) {
      if (d.tgt == nullptr || d.tgt_out == nullptr) {
        g_gemm_err = "target-logit epilogue: missing target pointers";
        return -2;
      }
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false)) return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_BF16_TGT>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the target-logit epilogue takes K-major operands and tiles of at least 128 columns";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_BF16_ROPE) {
    if constexpr (!A_MN && !B_MN) {
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false)) return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_BF16_ROPE>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the rotary epilogue takes K-major operands only";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_BF16_SWIGLU) {
    if constexpr (!A_MN && !B_MN) {
      CUtensorMap td;  // gate [M, N/2]: pieces of 32 rows x 64 columns
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false) ||
          !make_tmap(&td, d.aux, d.N / 2, d.M, d.ldaux, 64, 32, false))
        return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_BF16_SWIGLU>(ta, tb, tc, td, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the SwiGLU epilogue takes K-major operands only";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_BF16_RELU2) {
    if constexpr (!A_MN && !B_MN) {
      CUtensorMap td;  // gate [M, N], same pieces as C
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false) || !make_tmap(&td, d.aux, d.N, d.M, d.ldaux, 64, 32, false))
        return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_BF16_RELU2>(ta, tb, tc, td, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the ReLU^2 epilogue takes K-major operands only";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_CE_STATS || d.out == GEMM_OUT_CE_GRAD) {
    if constexpr (!A_MN && !B_MN && BN == 256 && (MT == 1 || MT == GEMM_MT_PAIR)) {
      if (d.out == GEMM_OUT_CE_STATS)  // no output tensor: the A map stands in for the unused descriptors
        return launch_tc<BN, MT, A_MN, B_MN, EPI_CE_STATS>(ta, tb, ta, ta, epi, d, whole, d_status, stream);
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false)) return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_CE_GRAD>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the classifier-head epilogues take K-major operands on 256-column tiles";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_DSWIGLU) {
    if constexpr (!A_MN && B_MN && ((BN == 256 && (MT == 1 || MT == GEMM_MT_PAIR)) || NARROW)) {
      CUtensorMap td;  // h13 in, d h13 out: [M, 2N] bf16, pieces of 32 rows x 64 columns
      if (!make_tmap(&tc, d.C, 2 * (uint64_t)d.N, d.M, d.ldc, 64, 32, false) ||
          !make_tmap(&td, d.aux, 2 * (uint64_t)d.N, d.M, d.ldaux, 64, 32, false))
        return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_DSWIGLU>(ta, tb, tc, td, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the SwiGLU-backward epilogue takes the dX form (A K-major, B MN-major) on 64- and 256-column tiles";
      return -2;
    }
  }
  if (d.out == GEMM_OUT_DRELU2) {
    if constexpr (!A_MN && B_MN && ((BN == 256 && (MT == 1 || MT == GEMM_MT_PAIR)) || NARROW)) {
      CUtensorMap td;  // h in, d h out: [M, N] bf16, pieces of 32 rows x 64 columns
      if (!make_tmap(&tc, d.C, d.N, d.M, d.ldc, 64, 32, false) || !make_tmap(&td, d.aux, d.N, d.M, d.ldaux, 64, 32, false))
        return -2;
      return launch_tc<BN, MT, A_MN, B_MN, EPI_DRELU2>(ta, tb, tc, td, epi, d, whole, d_status, stream);
    } else {
      g_gemm_err = "the ReLU^2-backward epilogue takes the dX form (A K-major, B MN-major) on 64- and 256-column tiles";
      return -2;
    }
  }
  }
  if (!make_tmap(&tc, d.C, d.N, d.part_rows > 0 ? (uint64_t)split_k * d.part_rows : d.M, d.ldc, 32, 32, true)) return -2;
  if (d.out == GEMM_OUT_F32) {
    if (d.part_rows > 0) return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_F32>(ta, tb, tc, tc, epi, d, split_k, d_status, stream);
    // One residual, K-major operands and room for the residual buffers: let TMA fetch the residual pieces.
    if constexpr (!A_MN && !B_MN && MT != GEMM_MT_PAIR2 && GemmCfg<BN, MT>::fits(EPI_STORE_F32_TMARES)) {
      static const bool no_tma_res = getenv("ANE_B200_NO_TMA_RES") != nullptr;  // A/B measurements
      if (d.res1 != nullptr && d.res2 == nullptr && !no_tma_res) {
        CUtensorMap td;
        if (!make_tmap(&td, d.res1, d.N, d.M, d.ldres, 32, 32, true)) return -2;
        return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_F32_TMARES>(ta, tb, tc, td, epi, d, whole, d_status, stream);
      }
    }
    return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_F32>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
  }
  if constexpr (GemmCfg<BN, MT>::PAIR || BN == 32) {
    g_gemm_err = "pair tiles and 32-column tiles are built for the non-accumulating epilogues";
    return -2;
  } else {
    if (d.first) return launch_tc<BN, MT, A_MN, B_MN, EPI_STORE_F32>(ta, tb, tc, tc, epi, d, whole, d_status, stream);
    return launch_tc<BN, MT, A_MN, B_MN, EPI_REDUCE_F32>(ta, tb, tc, tc, epi, d, split_k, d_status, stream);
  }
}

template <int BN, int MT>
static int dispatch_layout(const GemmDesc& d, int split_k, int* d_status, cudaStream_t stream) {
  CUtensorMap ta, tb;
  bool ok;
  // (hi | lo) operands: both halves of a row, and as many rows as there are
  const bool seg = d.seg_kb > 0;
  const int k_extent = seg ? 2 * d.seg_kb * GEMM_BK : d.K;
  if (!d.a_mn) ok = make_tmap(&ta, d.A, k_extent, d.M, d.lda, GEMM_BK, GEMM_BM);
  else         ok = make_tmap(&ta, d.A, seg ? d.lda : d.M, seg ? d.seg_k : d.K, d.lda, 64, GEMM_BK);
  if (!ok) return -2;
  // K-major B: one box per CTA and stage (a CTA of a pair loads half of the tile's rows)
  if (!d.b_mn) ok = make_tmap(&tb, d.B, k_extent, d.N, d.ldb, GEMM_BK, GemmCfg<BN, MT>::PAIR ? BN / 2 : BN);
  else         ok = make_tmap(&tb, d.B, seg ? d.ldb : d.N, seg ? d.seg_k : d.K, d.ldb, 64, GEMM_BK);
  if (!ok) return -2;
  if constexpr (BN == 32) {
    if (!d.a_mn && !d.b_mn) return dispatch_epi<BN, MT, false, false>(ta, tb, d, split_k, d_status, stream);
    g_gemm_err = "32-column tiles: unsupported operand layout";
    return -2;
  } else if constexpr (GemmCfg<BN, MT>::PAIR) {  // forward and dX forms only (A K-major)
    if (!d.a_mn && !d.b_mn) return dispatch_epi<BN, MT, false, false>(ta, tb, d, split_k, d_status, stream);
    if (!d.a_mn && d.b_mn) return dispatch_epi<BN, MT, false, true>(ta, tb, d, split_k, d_status, stream);
    g_gemm_err = "cluster tiles: unsupported operand layout";
    return -2;
  } else {
  if (!d.a_mn && !d.b_mn) return dispatch_epi<BN, MT, false, false>(ta, tb, d, split_k, d_status, stream);
  if (!d.a_mn && d.b_mn) return dispatch_epi<BN, MT, false, true>(ta, tb, d, split_k, d_status, stream);
  if (d.a_mn && d.b_mn) return dispatch_epi<BN, MT, true, true>(ta, tb, d, split_k, d_status, stream);
  return dispatch_epi<BN, MT, true, false>(ta, tb, d, split_k, d_status, stream);
  }
}

// ------------------------------------------------------------------------------------------
// Tile / schedule selection.
//   128-row tiles: width by a waves x width cost (wider tiles win unless they leave the last wave
//   mostly empty; 128-wide tiles stall on shared-memory fill); accumulating GEMMs take the width that
//   pads N least and classic split-K when it fills whole waves, else stream-K.
//   256-row tiles (two A sub-tiles share each B tile: a third less shared-memory fill per FLOP, but
//   no second TMEM accumulator set, so the epilogue is not hidden): measured faster by 5-15 % when
//   the main loop is long (K >= 2048), the 256-row tiles still cover most SMs and the epilogue is
//   short (no residual; M >= 2048 for weight gradients); slower otherwise.
// ------------------------------------------------------------------------------------------
struct GemmPlan {
  int bn = 256, mt = 1, sched = 1;  // sched > 0: classic persistent with that split-K; 0: stream-K
};

static GemmPlan plan_gemm(const GemmDesc& d, int sms) {
  const int kblocks = (d.K + GEMM_BK - 1) / GEMM_BK;
  static const int force_mt = [] {
    const char* e = getenv("ANE_B200_GEMM_MT");  // 1 or 2 pins the tile height (measurements)
    return e ? atoi(e) : 0;
  }();
  GemmPlan p;
  const bool accum = d.out == GEMM_OUT_ACCUM;
  // ---- 256-row tiles
  if (force_mt != 1 && d.M > 128 && (kblocks >= 32 || force_mt == 2)) {
    const int tiles_m2 = (d.M + 255) / 256;
    int bn2 = 256;
    long pad_best = -1;
    for (int bn : {256, 192}) {  // least padding of N, ties to the wider tile
      const long pad = (long)((d.N + bn - 1) / bn) * bn;
      if (pad_best < 0 || pad < pad_best) {
        pad_best = pad;
        bn2 = bn;
      }
    }
    const long tiles2 = (long)tiles_m2 * ((d.N + bn2 - 1) / bn2);
    if (accum && d.split_k <= 0 && (d.M >= 2048 || force_mt == 2)) {
      p.mt = 2;
      p.bn = bn2;
      int split = (int)(sms / tiles2);
      int max_split = kblocks / 4;
      if (max_split < 1) max_split = 1;
      if (split > max_split) split = max_split;
      if (split < 1) split = 1;
      const long waves = (tiles2 * split + sms - 1) / sms;
      const long classic_cost = waves * ((kblocks + split - 1) / split);
      const long streamk_cost = (tiles2 * kblocks + sms - 1) / sms + 8;
      p.sched = (streamk_cost < classic_cost && tiles2 * kblocks >= 8L * sms) ? 0 : split;
      return p;
    }
    if (!accum && ((d.res1 == nullptr && d.res2 == nullptr) || force_mt == 2)) {
      // whole waves only: a last wave that is mostly empty costs more than the fill saves; and no
      // residual epilogue, which is long and would no longer hide behind the next tile
      double best_eff = 0.0;
      int best_bn = 256;
      for (int bn : {256, 192}) {
        const long t = (long)tiles_m2 * ((d.N + bn - 1) / bn);
        const long waves = (t + sms - 1) / sms;
        const double eff = (double)t / (double)(waves * sms) * ((double)d.N / (double)(((d.N + bn - 1) / bn) * bn));
        if (eff > best_eff + 1e-9) {
          best_eff = eff;
          best_bn = bn;
        }
      }
      if (force_mt == 2 || best_eff >= 0.8) {
        p.mt = 2;
        p.bn = best_bn;
        p.sched = 1;
        return p;
      }
    }
  }
  // ---- 128-row tiles
  const int tiles_m = (d.M + GEMM_BM - 1) / GEMM_BM;
  if (accum && d.split_k <= 0) {
    int best_bn = 256;
    long best_pad = -1;
    for (int bn : {256, 192, 128}) {
      const long pad = (long)((d.N + bn - 1) / bn) * bn;
      if (best_pad < 0 || pad < best_pad) {
        best_pad = pad;
        best_bn = bn;
      }
    }
    const int tiles = tiles_m * ((d.N + best_bn - 1) / best_bn);
    int split = sms / tiles;
    int max_split = kblocks / 4;
    if (max_split < 1) max_split = 1;
    if (split > max_split) split = max_split;
    if (split < 1) split = 1;
    const long waves = ((long)tiles * split + sms - 1) / sms;
    const long classic_cost = waves * ((kblocks + split - 1) / split);
    const long streamk_cost = ((long)tiles * kblocks + sms - 1) / sms + 8;
    p.bn = best_bn;
    p.sched = (streamk_cost < classic_cost) ? 0 : split;
    return p;
  }
  long best_cost = -1;
  for (int bn : {256, 192, 128}) {
    const int tiles = tiles_m * ((d.N + bn - 1) / bn);
    const int split_k = accum ? d.split_k : 1;
    const long waves = ((long)tiles * split_k + sms - 1) / sms;
    const long kb = (kblocks + split_k - 1) / split_k;
    long cost = waves * kb * bn;
    if (bn == 128) cost += cost / 3;   // fill-rate penalty of the narrow tile
    if (bn == 192) cost += cost / 10;  // a narrower tile must win clearly
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      p.bn = bn;
      p.sched = split_k;
    }
  }
  return p;
}

// Clusters of `size` (2, 4 or 8) CTAs of the fp32 kernel, each with an SM's shared memory, that the device holds at once.
static int resident_clusters_f32(int size) {
  static int known[4] = {-1, -1, -1, -1};
  auto kern = gemm_f32_tc_kernel<true, true, true>;
  const int at = size == 8 ? 3 : size == 4 ? 2 : 1;
  if (known[at] < 0) {
    int n = 0;
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3((unsigned)(size * 148));
    q.blockDim = dim3(F32TC_THREADS);
    q.dynamicSmemBytes = F32TC_SMEM;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeClusterDimension;
    a[0].val.clusterDim.x = (unsigned)size;
    a[0].val.clusterDim.y = 1;
    a[0].val.clusterDim.z = 1;
    q.attrs = a;
    q.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F32TC_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &q) != cudaSuccess)
      n = 0;  // a part of a GPU may hold no cluster of this size: products take whole tiles there
    cudaGetLastError();
    known[at] = std::min(n, gemm_num_sms() / size);
  }
  return known[at];
}

// Width of a narrow tile (64 or 32 columns; 0: none) for a product with less than a wave of 128 x 128 tiles.  One CTA per SM
// then, and its time is that of its own chain: k-blocks of about 310 cycles at 32 columns, 330 at 64 and 370 at 128 (more SMs pull
// operands, each of them less), and an epilogue of about 700 cycles per staged piece, four of them for 128 fp32 columns.  Every
// element is the same sum in the same order whatever the width.  us, 128 columns -> narrow: 256 x 2304 x 768 (bf16) 6.2 -> 5.8,
// 256 x 768 x 768 (fp32 + residual) 8.8 -> 5.6, 256 x 768 x 2048 12.4 -> 9.0, 512 x 768 x 6144 26.0 -> 20.9, 1000 x 288 x 288 8.2 -> 4.4,
// accumulated 768 x 768 x 256 7.3 -> 5.0, 2304 x 768 x 440 (the line: eight k-blocks) 8.7 both, SwiGLU backward of 256 x 2048 x 768
// 9.2 -> 7.5; of 440 products of 48 to 2048 rows none was slower.
static int narrow_width(const GemmDesc& d) {
  static const bool off = [] { const char* e = getenv("ANE_B200_GEMM_NARROW"); return e && e[0] == '0'; }();  // A/B measurements
  if (off || d.split_k > 1) return 0;
  const bool f32 = d.out == GEMM_OUT_F32 || d.out == GEMM_OUT_ACCUM;
  if (!f32 && d.out != GEMM_OUT_DSWIGLU && d.out != GEMM_OUT_DRELU2 && d.out != GEMM_OUT_BF16 && d.out != GEMM_OUT_BF16_ROPE &&
      d.out != GEMM_OUT_BF16_SWIGLU && d.out != GEMM_OUT_BF16_RELU2)
    return 0;
  const int sms = gemm_num_sms();
  const long tiles_m = (d.M + GEMM_BM - 1) / GEMM_BM, kblocks = (d.K + GEMM_BK - 1) / GEMM_BK;
  if (tiles_m * ((d.N + 127) / 128) > sms) return 0;
  // weight gradients over eight k-blocks or more share out the contraction instead (plan_gemm)
  if (d.out == GEMM_OUT_ACCUM && kblocks >= 8) return 0;
  int best_bn = 0;
  long best = 0;
  for (int bn : {128, 64, 32}) {
    if (bn == 32 && (d.out != GEMM_OUT_F32 || d.a_mn || d.b_mn)) continue;
    const long waves = (tiles_m * ((d.N + bn - 1) / bn) + sms - 1) / sms;
    const long cost = waves * kblocks * (290 + 5 * bn / 8) + bn / (f32 || d.out == GEMM_OUT_DSWIGLU ? 32 : 64) * 700;
    if (best == 0 || cost < best) {
      best = cost;
      best_bn = bn;
    }
  }
  return best_bn < 128 ? best_bn : 0;
}
// Shares of the contraction for a product of few tiles whose consumer adds them up, and the tiles' width; 1: none.  The chain of one
// CTA is its k-blocks (see narrow_width); a share more costs the consumer about 300 cycles of reading.  us, whole -> shares: 256 x 768
// x 2304 13.3 -> 9.4, 256 x 768 x 4096 18.3 -> 10.1, 256 x 768 x 32000 96 -> 23, 512 x 768 x 32000 in three passes 285 -> 69, 1000 x
// 288 x 1536 11.2 -> 8.8, 1000 x 288 x 32000 98 -> 29; the norm behind them 5.3 -> 7.5 at six shares of 256 x 768, 4.0 -> 5.0 at
// three of 1000 x 288.  (In a pass: one window 2469 -> 2297 us an update, three micro-steps of 5 x 200 3030 -> 2812, the split-precision
// update of 2 x 256 6749 -> 6287.)  Against the fp32 engine the split-precision gradients are half as far off in shares, shorter chains
// of sums (2.1 to 3.6e-5 for 6.2 to 6.9e-5), and the bf16 ones as far (4.7 to 11.3e-3).
static int plan_parts(const GemmDesc& d, int& best_bn) {
  static const bool off = [] { const char* e = getenv("ANE_B200_GEMM_PARTS"); return e && e[0] == '0'; }();  // A/B measurements
  if (off || d.parts == nullptr || d.n_parts == nullptr || d.out != GEMM_OUT_F32 || d.res1 || d.res2 || d.split_k > 1 || d.N % 4 != 0 ||
      (reinterpret_cast<uintptr_t>(d.parts) & 15) != 0)
    return 1;
  const int sms = gemm_num_sms();
  const long tiles_m = (d.M + GEMM_BM - 1) / GEMM_BM, kblocks = (d.K + GEMM_BK - 1) / GEMM_BK;
  const size_t part = sizeof(float) * (size_t)parts_rows(d.M) * d.N;
  int best = 1;
  long least = 0;
  for (int bn : {64, 128}) {
    const long tiles = tiles_m * ((d.N + bn - 1) / bn);
    if (tiles > sms) continue;
    for (int most = 1; most <= kMostParts && tiles * most <= sms && (most == 1 || part * most <= d.parts_bytes); ++most) {
      const long share = (kblocks + most - 1) / most;
      const int n = (int)((kblocks + share - 1) / share);  // (none is empty)
      const long cost = share * (290 + 5 * bn / 8) + bn / 32 * 700 + (n > 1 ? 300 * n : 0);
      if (least == 0 || cost < least) {
        least = cost;
        best = n;
        best_bn = bn;
      }
    }
  }
  return best;
}
bool gemm_whole_tiles(const GemmDesc& d) {
  return d.out == GEMM_OUT_ACCUM && (narrow_width(d) != 0 || plan_gemm(d, gemm_num_sms()).sched == 1);
}
int gemm_bf16(const GemmDesc& d, int* d_status, cudaStream_t stream) {
  if (d.n_parts) *d.n_parts = 1;
  if (d.first && !gemm_whole_tiles(d)) {
    g_gemm_err = "a product in shares of the contraction adds to C and cannot overwrite it";
    return -2;
  }
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return 0;
  if (d.out == GEMM_OUT_F32 && (d.res1 || d.res2) && (d.ldres % 4 != 0 ||
      (reinterpret_cast<uintptr_t>(d.res1) & 15) != 0 || (reinterpret_cast<uintptr_t>(d.res2) & 15) != 0)) {
    g_gemm_err = "fp32 residual operands must be 16-byte aligned with ldres % 4 == 0";
    return -2;
  }
  if (d.out == GEMM_OUT_BF16_SWIGLU && (d.aux == nullptr || d.N % 128 != 0 || d.ldaux % 8 != 0 ||
                                        (reinterpret_cast<uintptr_t>(d.aux) & 15) != 0)) {
    g_gemm_err = "SwiGLU epilogue: N must be a multiple of 128 and the gate buffer 16-byte aligned with ldaux % 8 == 0";
    return -2;
  }
  if (d.out == GEMM_OUT_BF16_RELU2 && (d.aux == nullptr || d.ldaux % 8 != 0 || (reinterpret_cast<uintptr_t>(d.aux) & 15) != 0)) {
    g_gemm_err = "ReLU^2 epilogue: the gate buffer must be 16-byte aligned with ldaux % 8 == 0";
    return -2;
  }
  if (d.out == GEMM_OUT_BF16_ROPE &&
      (d.rope_cos == nullptr || d.rope_sin == nullptr || d.rope_seq <= 0 || d.rope_cols % 64 != 0 || d.alpha != 1.f ||
       (reinterpret_cast<uintptr_t>(d.rope_cos) & 15) != 0 || (reinterpret_cast<uintptr_t>(d.rope_sin) & 15) != 0)) {
    g_gemm_err = "rotary epilogue: needs 16-byte aligned cos/sin tables, rope_seq > 0, rope_cols % 64 == 0 and alpha == 1";
    return -2;
  }
  if (d.out == GEMM_OUT_DSWIGLU || d.out == GEMM_OUT_DRELU2) {
    if (d.aux == nullptr || d.a_mn || !d.b_mn || d.N % (d.out == GEMM_OUT_DRELU2 ? 64 : 32) != 0 || d.ldaux % 8 != 0 ||
        d.ldc % 8 != 0 || (reinterpret_cast<uintptr_t>(d.aux) & 15) != 0) {
      g_gemm_err = "SwiGLU / ReLU^2 backward epilogue: dX form only, N % 32 == 0 (ReLU^2: % 64), the saved activations and the "
                   "output 16-byte aligned with pitches % 8 == 0";
      return -2;
    }
    if (narrow_width(d) == 64) return dispatch_layout<64, 1>(d, 1, d_status, stream);
    // 256-column tiles: CTA pairs when they fill their waves (the step's shape), else one CTA per tile
    const int pairs = gemm_num_sms() / 2;
    const long tiles = (long)((d.M + 255) / 256) * ((d.N + 255) / 256);
    const long waves = (tiles + pairs - 1) / pairs;
    const double eff = (double)tiles / (double)(waves * pairs);
    static const bool no_pair = [] { const char* e = getenv("ANE_B200_GEMM_PAIR"); return e && atoi(e) == 0; }();
    if (!no_pair && d.M >= 256 && eff >= 0.8) return dispatch_layout<256, GEMM_MT_PAIR>(d, 1, d_status, stream);
    return dispatch_layout<256, 1>(d, 1, d_status, stream);
  }
  if (d.out == GEMM_OUT_CE_STATS || d.out == GEMM_OUT_CE_GRAD) {
    const bool stats = d.out == GEMM_OUT_CE_STATS;
    if (d.a_mn || d.b_mn || d.tgt == nullptr || (stats && (d.ce_stats == nullptr || d.tgt_out == nullptr || d.ce_rows < d.M)) ||
        (!stats && (d.ce_lse2 == nullptr || d.ce_coef == nullptr || d.C == nullptr))) {
      g_gemm_err = "classifier-head epilogue: K-major operands, targets and the statistics / per-row buffers are required";
      return -2;
    }
    const int pairs = gemm_num_sms() / 2;
    const long tiles = (long)((d.M + 255) / 256) * ((d.N + 255) / 256);
    const long waves = (tiles + pairs - 1) / pairs;
    const double eff = (double)tiles / (double)(waves * pairs);
    static const bool no_pair = [] { const char* e = getenv("ANE_B200_GEMM_PAIR"); return e && atoi(e) == 0; }();
    if (!no_pair && d.M >= 256 && eff >= 0.8) return dispatch_layout<256, GEMM_MT_PAIR>(d, 1, d_status, stream);
    return dispatch_layout<256, 1>(d, 1, d_status, stream);
  }
  int parts_bn = 0;
  if (const int n = plan_parts(d, parts_bn); n > 1) {
    GemmDesc e = d;
    e.C = d.parts;
    e.ldc = d.N;
    e.part_rows = parts_rows(d.M);
    *d.n_parts = n;
    return parts_bn == 64 ? dispatch_layout<64, 1>(e, n, d_status, stream) : dispatch_layout<128, 1>(e, n, d_status, stream);
  }
  if (const int bn = narrow_width(d))
    return bn == 64 ? dispatch_layout<64, 1>(d, 1, d_status, stream) : dispatch_layout<32, 1>(d, 1, d_status, stream);
  GemmPlan p = plan_gemm(d, gemm_num_sms());
  if (d.out == GEMM_OUT_BF16_SWIGLU && p.bn == 192) p.bn = 256;  // gate rows pair up two 64-column pieces
  // CTA-pair tiles (256 x 256 per two SMs, half of the B tile per CTA): measured faster than both single-CTA
  // forms when K is short (the 256-row single-CTA tile cannot hide its epilogue there) and the tiles fill the
  // pairs' waves; slower for N = 768 (96 tiles on 74 pairs) and for long K.
  static const int pair_env = [] {
    // 0: off; 128 | 192 | 256: 256-row pair tiles of that width, 512: 512 x 192 pair tiles, wherever pairs apply
    const char* e = getenv("ANE_B200_GEMM_PAIR");
    return e ? atoi(e) : -1;
  }();
  if (pair_env != 0 && d.out != GEMM_OUT_ACCUM && !d.a_mn && d.M >= 256) {
    int bn = 0;
    if (pair_env > 0) {
      bn = pair_env;
      if (bn == 192 && d.out == GEMM_OUT_BF16_SWIGLU) bn = 256;
    } else {
      const int pairs = gemm_num_sms() / 2;
      const long tiles = (long)((d.M + 255) / 256) * ((d.N + 255) / 256);
      const long waves = (tiles + pairs - 1) / pairs;
      const double eff = (double)tiles / (double)(waves * pairs) * ((double)d.N / (double)(((d.N + 255) / 256) * 256));
      const int kblocks = (d.K + GEMM_BK - 1) / GEMM_BK;
      if (kblocks < 32 && eff >= 0.85) {
        bn = 256;
      } else if (d.out != GEMM_OUT_BF16_SWIGLU) {
        // 512 x 192 tiles (two sub-tiles per CTA, one accumulator set): the least fill per FLOP.  For the
        // N = 768 shapes they make one wave of 64 tiles; measured faster than the single-CTA 256-row tile for
        // K >= 2048 and for the short-K bf16 store, slower for the short-K residual epilogue (which is exposed).
        const long tiles2 = (long)((d.M + 511) / 512) * ((d.N + 191) / 192);
        const long waves2 = (tiles2 + pairs - 1) / pairs;
        const double eff2 =
            (double)tiles2 / (double)(waves2 * pairs) * ((double)d.N / (double)(((d.N + 191) / 192) * 192));
        const bool residual = d.res1 != nullptr || d.res2 != nullptr;
        if (eff2 >= 0.85 && !(kblocks < 32 && residual)) bn = 512;
        // A long K with a residual that TMA can fetch: 256 x 192 tiles, whose first epilogues hide behind the tiles after them.  us, this
        // against what is chosen otherwise: 8192 x 768 x 2048 32.1 / 40.3, 8192 x 2304 x 2048 80 / 114, 16384 x 768 x 2048 64 / 82,
        // 12288 x 768 x 3072 62.7 / 62.3, 6144 x 512 x 2048 20.3 / 21.3 (34 products of 3000 to 16384 rows and K up to 3072: 0.99 to
        // 1.48 times as fast).  From K = 4096 on, in several waves, an epilogue is a small part and the wider tiles' fill counts: 12288 x 768 x
        // 4096 83 / 78, 8192 x 768 x 8192 96 / 86, 16384 x 768 x 8192 209 / 193.  In one wave these stay ahead: 4096 x 768 x 8192 45.6 / 52.1.
        const long tiles3 = (long)((d.M + 255) / 256) * ((d.N + 191) / 192);
        const double eff3 = (double)tiles3 / (double)((tiles3 + pairs - 1) / pairs * pairs) * ((double)d.N / (double)(((d.N + 191) / 192) * 192));
        if (kblocks >= 32 && (kblocks < 64 || tiles3 <= pairs) && d.res1 != nullptr && d.res2 == nullptr && !d.b_mn && eff3 >= 0.8) bn = 192;
      }
    }
    if (bn == 512 && d.out != GEMM_OUT_BF16_SWIGLU) return dispatch_layout<192, GEMM_MT_PAIR2>(d, 1, d_status, stream);
    if (bn == 256) return dispatch_layout<256, GEMM_MT_PAIR>(d, 1, d_status, stream);
    if (bn == 192) return dispatch_layout<192, GEMM_MT_PAIR>(d, 1, d_status, stream);
    if (bn == 128) return dispatch_layout<128, GEMM_MT_PAIR>(d, 1, d_status, stream);
  }
  if (p.mt == 2) {
    if (p.bn == 256) return dispatch_layout<256, 2>(d, p.sched, d_status, stream);
    return dispatch_layout<192, 2>(d, p.sched, d_status, stream);
  }
  if (p.bn == 256) return dispatch_layout<256, 1>(d, p.sched, d_status, stream);
  if (p.bn == 192) return dispatch_layout<192, 1>(d, p.sched, d_status, stream);
  return dispatch_layout<128, 1>(d, p.sched, d_status, stream);
}

// ------------------------------------------------------------------------------------------
// Grouped accumulating products: C_p += A_p^T B_p for up to four problems with one contraction length, both
// operands stored [K, .] (the weight gradients of a layer), one stream-K launch over the concatenated tiles
// of 256 x 256.  `slot` is device memory for the group's descriptors; it is filled on the first call for a
// given slot (`*built`) and reused afterwards -- the operands of a layer never move.
// ------------------------------------------------------------------------------------------
int gemm_bf16_grouped(const GemmDesc* ds, int n, void* slot, bool* built, int* d_status, cudaStream_t stream) {
  if (n < 1 || n > 4 || slot == nullptr || built == nullptr) {
    g_gemm_err = "grouped GEMM: one to four problems and a descriptor slot are required";
    return -2;
  }
  constexpr int BN = 256, MT = 2;
  constexpr int BM_TILE = GemmCfg<BN, MT>::BM_TILE;
  int K = ds[0].K;
  long tiles = 0;
  for (int p = 0; p < n; ++p) {
    const GemmDesc& d = ds[p];
    if (!d.a_mn || !d.b_mn || d.out != GEMM_OUT_ACCUM || d.K != K || d.alpha != 1.f || d.M <= 0 || d.N <= 0) {
      g_gemm_err = "grouped GEMM: every problem must be C += A^T B with MN-major operands, alpha 1 and the same K";
      return -2;
    }
    tiles += (long)((d.M + BM_TILE - 1) / BM_TILE) * ((d.N + BN - 1) / BN);
  }
  if (!*built) {
    GemmGroup g;
    memset(&g, 0, sizeof g);
    g.n = n;
    int t0 = 0;
    for (int p = 0; p < n; ++p) {
      const GemmDesc& d = ds[p];
      if (!make_tmap(&g.a[p], d.A, d.M, d.K, d.lda, 64, GEMM_BK) || !make_tmap(&g.b[p], d.B, d.N, d.K, d.ldb, 64, GEMM_BK) ||
          !make_tmap(&g.c[p], d.C, d.N, d.M, d.ldc, 32, 32, true))
        return -2;
      g.M[p] = d.M;
      g.N[p] = d.N;
      g.tile0[p] = t0;
      t0 += ((d.M + BM_TILE - 1) / BM_TILE) * ((d.N + BN - 1) / BN);
    }
    g.tile0[n] = t0;
    // synchronous copy: the descriptors must be in place before the launch below and the source is on the stack
    if (cudaMemcpy(slot, &g, sizeof g, cudaMemcpyHostToDevice) != cudaSuccess) {
      g_gemm_err = "grouped GEMM: descriptor upload failed";
      return -3;
    }
    *built = true;
  }
  auto kern = gemm_tc_kernel<BN, MT, true, true, EPI_REDUCE_F32>;
  constexpr uint32_t smem_bytes = GemmCfg<BN, MT>::smem_bytes(EPI_REDUCE_F32);
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes) != cudaSuccess) {
      g_gemm_err = "grouped GEMM: cudaFuncSetAttribute failed";
      return -3;
    }
    attr_set = true;
  }
  const long long units = (long long)tiles * ((K + GEMM_BK - 1) / GEMM_BK);
  long long grid = units / 8;
  if (grid > gemm_num_sms()) grid = gemm_num_sms();
  if (grid < 1) grid = 1;
  CUtensorMap ta, tb, tc;  // the kernel's own map parameters are not used by a grouped launch; any valid maps do
  const GemmDesc& d0 = ds[0];
  if (!make_tmap(&ta, d0.A, d0.M, d0.K, d0.lda, 64, GEMM_BK) || !make_tmap(&tb, d0.B, d0.N, d0.K, d0.ldb, 64, GEMM_BK) ||
      !make_tmap(&tc, d0.C, d0.N, d0.M, d0.ldc, 32, 32, true))
    return -2;
  EpiParams epi{};
  epi.alpha = 1.f;
  cudaError_t e = launch_pdl(kern, dim3((unsigned)grid), dim3(GEMM_THREADS), smem_bytes, stream, ta, tb, tc, tc, epi, d0.M, d0.N,
                             K, 0, d_status, reinterpret_cast<const GemmGroup*>(slot));
  if (e != cudaSuccess) {
    g_gemm_err = std::string("grouped GEMM launch: ") + cudaGetErrorString(e);
    return -4;
  }
  return 0;
}
size_t gemm_group_slot_bytes() { return sizeof(GemmGroup); }

// ------------------------------------------------------------------------------------------
// Split-precision GEMM: fp32 operands as bf16 (hi, lo) pairs, three tensor-core products.
// ------------------------------------------------------------------------------------------
// Both operands of a product in one launch (blockIdx.y), four values per thread and step.  Operand [rows, cols] fp32
// with row pitch ld.  Two parts (hi, lo) lie beside one another in each row, [rows][hi (kp) | lo (kp)], kp = cols rounded up to 64,
// whichever way a product contracts: what has been cut for one serves the others (up to 8 where it is cut for one that contracts over
// rows alone).  Three (hi, mid, lo) lie behind one another along
// the contraction: for a K-major operand (k = cols) [rows][hi (kp) | mid | lo], for an MN-major one (k = rows) [hi (kp rows) | mid |
// lo][cols rounded up to 8], kp = k rounded up to a whole k-block.  What lies past cols, or k, is zero.  Three parts are exactly F32TC_SCALE times the fp32 value; where that is not
// finite, or its first part is not, the others are not either.
struct SplitOperand {
  const float* src;
  bf16* dst;
  long long ld;
  int rows, cols, kp, pitch, k_major, vec;  // vec: float4 reads are aligned
};
template <int PARTS>
__global__ void split_operands_kernel(const SplitOperand a, const SplitOperand b) {
  pdl_trigger();
  pdl_wait();
  const SplitOperand& o = blockIdx.y == 0 ? a : b;
  const int out_rows = o.k_major ? o.rows : o.kp, out_cols = o.k_major ? o.kp : o.pitch, per = out_cols / 4;
  const size_t next = o.k_major ? (size_t)o.kp : (size_t)o.kp * o.pitch;
  const long long total = (long long)out_rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int r = total <= 0xFFFFFFFFll ? (int)((unsigned)i / (unsigned)per) : (int)(i / per), c = (int)(i - (long long)r * per) * 4;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < o.rows) {
      const float* p = o.src + (size_t)r * o.ld + c;
      if (o.vec && c + 4 <= o.cols) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c + e < o.cols) x[e] = p[e];
      }
    }
    if constexpr (PARTS == 3) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] *= F32TC_SCALE;
    }
    bf16* q = o.dst + (size_t)r * o.pitch + c;
#pragma unroll
    for (int p = 0; p < PARTS; ++p, q += next) {
      __nv_bfloat162 v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        v[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
        x[2 * e] -= __bfloat162float(v[e].x);
        x[2 * e + 1] -= __bfloat162float(v[e].y);
      }
      *reinterpret_cast<uint2*>(q) = make_uint2(*reinterpret_cast<const uint32_t*>(&v[0]), *reinterpret_cast<const uint32_t*>(&v[1]));
    }
  }
}

bool SplitScratch::reserve(const size_t (&bytes)[2]) {
  for (int i = 0; i < 2; ++i) {
    if (cap[i] >= bytes[i]) continue;
    ++generation;
    if (buf[i]) cudaFree(buf[i]);
    buf[i] = nullptr;
    cap[i] = 0;
    if (cudaMalloc(&buf[i], bytes[i]) != cudaSuccess) {
      cudaGetLastError();
      buf[i] = nullptr;
      release();
      return false;
    }
    cap[i] = bytes[i];
  }
  return true;
}
int SplitScratch::grow(int i, size_t need, cudaStream_t stream) {
  if (cap[i] >= need) return 0;
  ++generation;
  // the previous, smaller buffer may still be read by GEMMs in flight on this stream
  if (buf[i]) {
    cudaStreamSynchronize(stream);
    cudaFree(buf[i]);
    buf[i] = nullptr;
    cap[i] = 0;
  }
  const size_t bytes = need + need / 4 + 256;
  if (cudaMalloc(&buf[i], bytes) != cudaSuccess) {
    cudaGetLastError();
    g_gemm_err = "split-precision GEMM: out of memory for the operands' parts";
    return GEMM_NO_SCRATCH;
  }
  cap[i] = bytes;
  return 0;
}
void SplitScratch::release() {
  if (buf[0] || buf[1]) ++generation;
  for (int i = 0; i < 2; ++i) {
    if (buf[i]) cudaFree(buf[i]);
    buf[i] = nullptr;
    cap[i] = 0;
  }
}

// Bytes of operand `i` of `d` in three bf16 parts, and their pitch.
static size_t parts_bytes(const GemmDesc& d, int i, int* pitch) {
  constexpr int parts = 3;
  const bool mn = i == 0 ? d.a_mn : d.b_mn;
  const int outer = i == 0 ? d.M : d.N, kp = (d.K + GEMM_BK - 1) / GEMM_BK * GEMM_BK;
  *pitch = mn ? (outer + 7) / 8 * 8 : parts * kp;
  return sizeof(bf16) * (size_t)(mn ? parts * kp : outer) * *pitch;
}
// The operands of `d` in three bf16 parts each, in the scratch.
static int split_operands(const GemmDesc& d, SplitScratch* sc, SplitOperand (&o)[2], cudaStream_t stream) {
  const int kp = (d.K + GEMM_BK - 1) / GEMM_BK * GEMM_BK;
  size_t used = 0;  // of an arena
  for (int i = 0; i < 2; ++i) {
    const bool mn = i == 0 ? d.a_mn : d.b_mn;
    const int outer = i == 0 ? d.M : d.N;
    o[i].src = reinterpret_cast<const float*>(i == 0 ? d.A : d.B);
    o[i].ld = i == 0 ? d.lda : d.ldb;
    o[i].rows = mn ? d.K : outer;
    o[i].cols = mn ? outer : d.K;
    o[i].kp = kp;
    o[i].k_major = mn ? 0 : 1;
    const size_t need = parts_bytes(d, i, &o[i].pitch);
    o[i].vec = o[i].ld % 4 == 0 && (reinterpret_cast<uintptr_t>(o[i].src) & 15) == 0;
    if (sc->arena != nullptr) {
      o[i].dst = reinterpret_cast<bf16*>(static_cast<char*>(sc->arena) + used);
      used += (need + 255) / 256 * 256;
      if (used > sc->arena_bytes) {
        g_gemm_err = "split-precision GEMM: the operands' parts do not fit the arena";
        return GEMM_NO_SCRATCH;
      }
      continue;
    }
    if (sc->cap[i] < need) return GEMM_NO_SCRATCH;
    o[i].dst = reinterpret_cast<bf16*>(sc->buf[i]);
  }
  const long long most = std::max((long long)(o[0].k_major ? o[0].rows : kp) * (o[0].k_major ? kp : o[0].pitch),
                                  (long long)(o[1].k_major ? o[1].rows : kp) * (o[1].k_major ? kp : o[1].pitch));
  const unsigned blocks = (unsigned)std::min<long long>(148 * 8, (most / 4 + 255) / 256);
  const cudaError_t e = launch_pdl(split_operands_kernel<3>, dim3(blocks, 2), dim3(256), 0, stream, o[0], o[1]);
  if (e != cudaSuccess) {
    g_gemm_err = "split-precision GEMM: operand split launch failed";
    return -4;
  }
  return 0;
}

// The three products run as one: its contraction is three passes of kp over (hi, lo), (lo, hi) and (hi, hi), so the
// accumulators stay in tensor memory between them; the small cross terms come first, while the accumulators are small too.  (Three launches, the second and third adding to C in memory, and
// two scalar conversion launches before them took 9.8 us each for 512 token rows.)
int gemm_bf16x3(const GemmDesc& d, SplitScratch* sc, int* d_status, cudaStream_t stream) {
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return 0;
  if (d.out != GEMM_OUT_F32 && d.out != GEMM_OUT_ACCUM) {
    g_gemm_err = "split-precision GEMM writes fp32 (store or accumulate) only";
    return -2;
  }
  SplitOperand cut[2];
  bf16* halves[2] = {static_cast<bf16*>(d.a_halves), static_cast<bf16*>(d.b_halves)};
  int pitch[2], cuts = 0;
  long long most = 0;
  for (int i = 0; i < 2; ++i) {
    const bool mn = i == 0 ? d.a_mn : d.b_mn;
    const int outer = i == 0 ? d.M : d.N, rows = mn ? d.K : outer, cols = mn ? outer : d.K;
    // (an operand of few columns that contracts over its rows would be up to eight times as wide in whole k-blocks)
    pitch[i] = mn && halves[i] == nullptr ? (cols + 7) / 8 * 16 : halves_pitch(cols);
    if (halves[i] != nullptr && (i == 0 ? d.a_cut : d.b_cut)) continue;
    if (halves[i] == nullptr) {
      if (const int rc = sc->grow(i, sizeof(bf16) * (size_t)rows * pitch[i], stream); rc != 0) return rc;
      halves[i] = reinterpret_cast<bf16*>(sc->buf[i]);
    }
    SplitOperand& o = cut[cuts++];
    o.src = reinterpret_cast<const float*>(i == 0 ? d.A : d.B);
    o.dst = halves[i];
    o.ld = i == 0 ? d.lda : d.ldb;
    o.rows = rows;
    o.cols = cols;
    o.kp = pitch[i] / 2;
    o.pitch = pitch[i];
    o.k_major = 1;
    o.vec = o.ld % 4 == 0 && (reinterpret_cast<uintptr_t>(o.src) & 15) == 0;
    most = std::max(most, (long long)rows * o.kp);
  }
  if (cuts > 0) {
    const unsigned blocks = (unsigned)std::min<long long>(148 * 8, (most / 4 + 255) / 256);
    if (launch_pdl(split_operands_kernel<2>, dim3(blocks, cuts), dim3(256), 0, stream, cut[0], cut[cuts - 1]) != cudaSuccess) {
      g_gemm_err = "split-precision GEMM: operand split launch failed";
      return -4;
    }
  }
  const int kp = (d.K + GEMM_BK - 1) / GEMM_BK * GEMM_BK;
  GemmDesc g = d;
  g.A = halves[0]; g.B = halves[1]; g.lda = pitch[0]; g.ldb = pitch[1];
  g.K = 3 * kp;
  g.seg_kb = kp / GEMM_BK;
  g.seg_k = d.K;
  return gemm_bf16(g, d_status, stream);
}

// ------------------------------------------------------------------------------------------
// fp32 GEMM on the FMA units (the fp32 mode).  Tiles of 16 TM x 16 TN, 256 threads with TM x TN accumulators each,
// a three-stage cp.async ring of 16-deep slices, two blocks per SM.
//   * Operands stay in the order they have in memory: K-major rows [m][k] with a pitch of 20 floats, MN-major slices
//     [k][m].  Either way four k of a thread's TM (TN) rows are TM (TN) conflict-free 16-byte reads, 4 TM TN FMAs for
//     TM + TN reads, so the FMA pipe is the limit (148 SMs x 128 FMA/clk: 72 TFLOP/s at 1.9 GHz).
//   * Few tiles (N = 288: 48 of 128 x 96) leave SMs idle, so the contraction is split over the blocks of a cluster;
//     their partial tiles meet in distributed shared memory, each block finishing a share of the rows: no workspace,
//     no atomics, always the same order of additions.
// The 64 x 64 kernel below (4 x 4 accumulators, scalar loads) took 327 us for 2048 x 288 x 288 with N tiles of 64.
// ------------------------------------------------------------------------------------------
static constexpr int F32_BK = 16, F32_STAGES = 3, F32_KPITCH = F32_BK + 4;

__device__ __forceinline__ void f32_copy16(uint32_t dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// One 16-deep slice of an operand's R rows: K-major [row][k] or MN-major [k][row].
template <int R, bool MN>
__device__ __forceinline__ void f32_load(uint32_t dst, const float* p, int row0, int rows, int k0, int k_end, int ld) {
  constexpr int CHUNKS = R * F32_BK / 4;
#pragma unroll
  for (int i = 0; i < (CHUNKS + 255) / 256; ++i) {
    const int c = threadIdx.x + i * 256;
    if (CHUNKS % 256 != 0 && c >= CHUNKS) break;
    if constexpr (MN) {
      const int k = c / (R / 4), r = (c - k * (R / 4)) * 4;
      const bool in = k0 + k < k_end && row0 + r < rows;
      f32_copy16(dst + (k * R + r) * 4, in ? p + (size_t)(k0 + k) * ld + row0 + r : p, in);
    } else {
      const int r = c >> 2, k = (c & 3) * 4;
      const bool in = k0 + k < k_end && row0 + r < rows;
      f32_copy16(dst + (r * F32_KPITCH + k) * 4, in ? p + (size_t)(row0 + r) * ld + k0 + k : p, in);
    }
  }
}
// f[i][q]: element k = 4 kk + q of this thread's row i
template <int T, bool MN>
__device__ __forceinline__ void f32_frag(float (&f)[T][4], const float* s, int kk, int t) {
  if constexpr (MN) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float* row = s + (4 * kk + q) * (16 * T);
      const float4 a = *reinterpret_cast<const float4*>(row + 4 * t);
      f[0][q] = a.x; f[1][q] = a.y; f[2][q] = a.z; f[3][q] = a.w;
      if constexpr (T == 8) {
        const float4 b = *reinterpret_cast<const float4*>(row + 64 + 4 * t);
        f[4][q] = b.x; f[5][q] = b.y; f[6][q] = b.z; f[7][q] = b.w;
      } else {
        const float2 b = *reinterpret_cast<const float2*>(row + 64 + 2 * t);
        f[4][q] = b.x; f[5][q] = b.y;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < T; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(s + (t + 16 * i) * F32_KPITCH + 4 * kk);
      f[i][0] = a.x; f[i][1] = a.y; f[i][2] = a.z; f[i][3] = a.w;
    }
  }
}
template <int T, bool MN>
__device__ __forceinline__ int f32_row(int t, int i) {  // tile row (column) of accumulator index i
  if (!MN) return t + 16 * i;
  if (i < 4) return 4 * t + i;
  return T == 8 ? 64 + 4 * t + (i - 4) : 64 + 2 * t + (i - 4);
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

struct F32Args {
  const float *A, *B;
  float* C;
  int M, N, K, lda, ldb, ldc, out, ldres, split, tiles_m;
  float alpha;
  const float *res1, *s1, *res2, *s2;
};

template <int TM, int TN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(256, 2) gemm_f32_tile_kernel(const F32Args a) {
  constexpr int BM = 16 * TM, BN = 16 * TN, A_FL = BM * F32_KPITCH, B_FL = BN * F32_KPITCH, CP = BN + 4;
  extern __shared__ __align__(16) float f32_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
  const int tile = blockIdx.x / a.split, rank = blockIdx.x - tile * a.split;
  const int m0 = (tile % a.tiles_m) * BM, n0 = (tile / a.tiles_m) * BN;
  const int slices = (a.K + F32_BK - 1) / F32_BK, per = (slices + a.split - 1) / a.split;
  const int k_begin = rank * per * F32_BK, k_end = min(a.K, k_begin + per * F32_BK);
  const int n_it = k_end > k_begin ? (k_end - k_begin + F32_BK - 1) / F32_BK : 0;
  const uint32_t sa = smem_u32(f32_smem), sb = sa + F32_STAGES * A_FL * 4;
  auto request = [&](int it) {
    if (it < n_it) {
      const int st = it % F32_STAGES, k0 = k_begin + it * F32_BK;
      f32_load<BM, A_MN>(sa + st * A_FL * 4, a.A, m0, a.M, k0, k_end, a.lda);
      f32_load<BN, B_MN>(sb + st * B_FL * 4, a.B, n0, a.N, k0, k_end, a.ldb);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  request(0);
  request(1);
  for (int it = 0; it < n_it; ++it) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    request(it + 2);  // its slot was read in iteration it - 1
    const float* As = f32_smem + (it % F32_STAGES) * A_FL;
    const float* Bs = f32_smem + F32_STAGES * A_FL + (it % F32_STAGES) * B_FL;
#pragma unroll
    for (int kk = 0; kk < F32_BK / 4; ++kk) {
      float fb[TN][4], fa[TM][4];
      f32_frag<TN, B_MN>(fb, Bs, kk, tx);
      f32_frag<TM, A_MN>(fa, As, kk, ty);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(fa[i][q], fb[j][q], acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) f32_smem[f32_row<TM, A_MN>(ty, i) * CP + f32_row<TN, B_MN>(tx, j)] = acc[i][j];
  if (a.split > 1) cluster_sync_all();
  else __syncthreads();
  float a1 = 0.f, a2 = 0.f;
  if (a.res1) a1 = a.s1 ? *a.s1 : 1.f;
  if (a.res2) a2 = a.s2 ? *a.s2 : 1.f;
  const int r0 = BM * rank / a.split, r1 = BM * (rank + 1) / a.split;
  for (int e = threadIdx.x; e < (r1 - r0) * (BN / 4); e += 256) {
    const int r = r0 + e / (BN / 4), c = (e % (BN / 4)) * 4, m = m0 + r, n = n0 + c;
    if (m >= a.M || n >= a.N) continue;
    const uint32_t at = sa + (uint32_t)(r * CP + c) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.split > 1) {
      for (int p = 0; p < a.split; ++p) {
        const float4 t = ld_cluster4(map_to_cta(at, p));
        v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
      }
    } else {
      v = *reinterpret_cast<const float4*>(f32_smem + r * CP + c);
    }
    v.x *= a.alpha; v.y *= a.alpha; v.z *= a.alpha; v.w *= a.alpha;
    float4* cp = reinterpret_cast<float4*>(a.C + (size_t)m * a.ldc + n);
    if (a.out == GEMM_OUT_ACCUM) {
      const float4 t = *cp;
      v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
    } else {
      if (a.res1) {
        const float4 t = *reinterpret_cast<const float4*>(a.res1 + (size_t)m * a.ldres + n);
        v.x += a1 * t.x; v.y += a1 * t.y; v.z += a1 * t.z; v.w += a1 * t.w;
      }
      if (a.res2) {
        const float4 t = *reinterpret_cast<const float4*>(a.res2 + (size_t)m * a.ldres + n);
        v.x += a2 * t.x; v.y += a2 * t.y; v.z += a2 * t.z; v.w += a2 * t.w;
      }
    }
    *cp = v;
  }
  if (a.split > 1) cluster_sync_all();  // the peers have read this block's partial sums
}

template <int TM, int TN, bool A_MN, bool B_MN>
static cudaError_t launch_f32_tile(const F32Args& a, int tiles, cudaStream_t stream) {
  auto kern = gemm_f32_tile_kernel<TM, TN, A_MN, B_MN>;
  constexpr size_t ring = sizeof(float) * F32_STAGES * (16 * TM + 16 * TN) * F32_KPITCH, out = sizeof(float) * 16 * TM * (16 * TN + 4);
  constexpr size_t bytes = ring > out ? ring : out;
  static unsigned long long done = 0;
  if (!smem_opt_in(kern, bytes, done)) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * a.split));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)a.split;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = a.split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, a);
}
template <int TM, int TN>
static cudaError_t launch_f32_layout(const F32Args& a, bool a_mn, bool b_mn, int tiles, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_f32_tile<TM, TN, false, false>(a, tiles, stream);
  if (!a_mn) return launch_f32_tile<TM, TN, false, true>(a, tiles, stream);
  if (b_mn) return launch_f32_tile<TM, TN, true, true>(a, tiles, stream);
  return launch_f32_tile<TM, TN, true, false>(a, tiles, stream);
}

// Tile and split: the fewest slice-times of the busiest SM (two blocks share one), counting padding and a start and
// end of about four slices per block; 96-wide tiles read more operands per FMA and must win by their padding.
static cudaError_t launch_f32(const GemmDesc& d, cudaStream_t stream) {
  const int slots = 2 * gemm_num_sms(), slices = (d.K + F32_BK - 1) / F32_BK;
  double best = 0;
  int bm = 8, bn = 8, split = 1;
  for (int tm : {8, 6})
    for (int tn : {8, 6})
      for (int sp : {1, 2, 4, 8}) {
        if (sp > 1 && sp * 2 > slices) continue;
        const long tiles = (long)((d.M + 16 * tm - 1) / (16 * tm)) * ((d.N + 16 * tn - 1) / (16 * tn));
        const long waves = (tiles * sp + slots - 1) / slots;
        const double pen = tm + tn == 16 ? 1.0 : tm + tn == 14 ? 1.05 : 1.1;
        const double cost = (double)waves * (((slices + sp - 1) / sp) + 4 + (sp > 1 ? 2 : 0)) * tm * tn * pen;
        if (best == 0 || cost < best) {
          best = cost;
          bm = tm;
          bn = tn;
          split = sp;
        }
      }
  F32Args a{reinterpret_cast<const float*>(d.A), reinterpret_cast<const float*>(d.B), reinterpret_cast<float*>(d.C), d.M, d.N, d.K, d.lda, d.ldb,
            d.ldc, d.out, d.ldres, split, (d.M + 16 * bm - 1) / (16 * bm), d.alpha, d.res1, d.s1, d.res2, d.s2};
  const int tiles = a.tiles_m * ((d.N + 16 * bn - 1) / (16 * bn));
  if (bm == 8 && bn == 8) return launch_f32_layout<8, 8>(a, d.a_mn, d.b_mn, tiles, stream);
  if (bm == 8) return launch_f32_layout<8, 6>(a, d.a_mn, d.b_mn, tiles, stream);
  if (bn == 8) return launch_f32_layout<6, 8>(a, d.a_mn, d.b_mn, tiles, stream);
  return launch_f32_layout<6, 6>(a, d.a_mn, d.b_mn, tiles, stream);
}
// What the 16-byte copies of the tiled kernel need.
static bool f32_aligned(const GemmDesc& d) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return al(d.A) && al(d.B) && al(d.C) && al(d.res1) && al(d.res2) && d.lda % 4 == 0 && d.ldb % 4 == 0 && d.ldc % 4 == 0 && d.N % 4 == 0 &&
         (!(d.res1 || d.res2) || d.ldres % 4 == 0) && (d.a_mn ? d.M % 4 == 0 : d.K % 4 == 0) && (d.b_mn || d.K % 4 == 0);
}

// ------------------------------------------------------------------------------------------
// The same for operands that are not 16-byte aligned: 64x64x16 tiles, 256 threads, 4x4 micro-tiles.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N,
                int K, int lda, int ldb, int ldc, int a_mn, int b_mn, int out, float alpha,
                const float* __restrict__ res1, const float* __restrict__ s1, const float* __restrict__ res2,
                const float* __restrict__ s2, int ldres) {
  __shared__ float As[16][65];
  __shared__ float Bs[16][65];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += 16) {
    for (int idx = threadIdx.x; idx < 64 * 16; idx += 256) {
      int kk, mm;
      if (a_mn) { mm = idx & 63; kk = idx >> 6; } else { kk = idx & 15; mm = idx >> 4; }
      const int gm = m0 + mm, gk = k0 + kk;
      float v = 0.f;
      if (gm < M && gk < K) v = a_mn ? A[(size_t)gk * lda + gm] : A[(size_t)gm * lda + gk];
      As[kk][mm] = v;
      int nn;
      if (b_mn) { nn = idx & 63; kk = idx >> 6; } else { kk = idx & 15; nn = idx >> 4; }
      const int gn = n0 + nn;
      const int gk2 = k0 + kk;
      v = 0.f;
      if (gn < N && gk2 < K) v = b_mn ? B[(size_t)gk2 * ldb + gn] : B[(size_t)gn * ldb + gk2];
      Bs[kk][nn] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  float a1 = 0.f, a2 = 0.f;
  if (res1) a1 = s1 ? *s1 : 1.f;
  if (res2) a2 = s2 ? *s2 : 1.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = alpha * acc[i][j];
      if (out == GEMM_OUT_ACCUM) {
        C[(size_t)m * ldc + n] += v;
      } else {
        if (res1) v += a1 * res1[(size_t)m * ldres + n];
        if (res2) v += a2 * res2[(size_t)m * ldres + n];
        C[(size_t)m * ldc + n] = v;
      }
    }
  }
}

// CTAs per tile of the tensor-core form: what gives the shortest chain, counting a start and end of about two k-blocks and two
// more for the exchange; 0: the FMA kernels are faster (or have to take it).
static int f32_on_tensor_cores(const GemmDesc& d) {
  static const bool off = [] { const char* e = getenv("ANE_B200_F32_TC"); return e && e[0] == '0'; }();  // A/B measurements
  if (off || !f32_aligned(d) || d.K < 128 || (d.out != GEMM_OUT_F32 && d.out != GEMM_OUT_ACCUM)) return 0;
  const int sms = gemm_num_sms();
  const long tiles = (long)((d.M + 127) / 128) * ((d.N + 127) / 128), kblocks = (d.K + GEMM_BK - 1) / GEMM_BK;
  long best = 0;
  int parts = 1;
  for (int p : {1, 2, 4, 8}) {
    if (p > 1 && (kblocks < 2 * p || tiles > resident_clusters_f32(p))) continue;
    const long cost = (tiles * p + sms - 1) / sms * ((kblocks + p - 1) / p) + 2 + (p > 1 ? 2 : 0);
    if (best == 0 || cost < best) {
      best = cost;
      parts = p;
    }
  }
  // us: k-blocks at 1.25, the cut (4 bytes read, 6 written per element) and its launch; the FMA kernels at about 40 TFLOP/s.  Of 176
  // products of 64 to 4096 rows, all layouts, those that this sends to the tensor cores are 1.28 to 5.1 times as fast there: next to
  // the line 768 x 768 x 256 12.9 us (16.5 on the FMA units), 768 x 768 x 512 17.3 (22.7), 512 x 1536 x 288 14.5 (22.7), 1024 x 288 x
  // 768 14.2 (20.6).  The other side may be up to 1.4 times too slow: 256 x 768 x 768 takes 20.6 where 400 x 768 x 768 takes 14.3.
  const double tc = 1.25 * best + ((double)d.M + d.N) * d.K * 10.0 / 5e6 + 4.0, fma = 2.0 * d.M * d.N * d.K / 40e6 + 5.0;
  return tc < fma ? parts : 0;
}

template <bool A_MN, bool B_MN, bool SPLIT>
static bool load_f32_tc() {
  static unsigned long long done = 0;
  return smem_opt_in(gemm_f32_tc_kernel<A_MN, B_MN, SPLIT>, F32TC_SMEM, done);
}
template <bool A_MN, bool B_MN, bool SPLIT>
static cudaError_t launch_f32_tc(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const F32TcArgs& a, int* d_status, cudaStream_t stream) {
  auto kern = gemm_f32_tc_kernel<A_MN, B_MN, SPLIT>;
  if (!load_f32_tc<A_MN, B_MN, SPLIT>()) return cudaErrorInvalidValue;
  const int tiles = ((a.M + 127) / 128) * ((a.N + 127) / 128);
  if constexpr (SPLIT)
    return launch_pdl_cluster(kern, dim3((unsigned)(tiles * a.parts)), dim3(F32TC_THREADS), F32TC_SMEM, stream, (unsigned)a.parts, ta, tb, tc, a, d_status);
  else
    return launch_pdl(kern, dim3((unsigned)std::min(tiles, gemm_num_sms())), dim3(F32TC_THREADS), F32TC_SMEM, stream, ta, tb, tc, a, d_status);
}
template <bool SPLIT>
static cudaError_t launch_f32_tc_layout(const GemmDesc& d, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const F32TcArgs& a, int* d_status, cudaStream_t stream) {
  if (!d.a_mn && !d.b_mn) return launch_f32_tc<false, false, SPLIT>(ta, tb, tc, a, d_status, stream);
  if (!d.a_mn) return launch_f32_tc<false, true, SPLIT>(ta, tb, tc, a, d_status, stream);
  if (d.b_mn) return launch_f32_tc<true, true, SPLIT>(ta, tb, tc, a, d_status, stream);
  return launch_f32_tc<true, false, SPLIT>(ta, tb, tc, a, d_status, stream);
}
static int gemm_f32_tc(const GemmDesc& d, int parts, SplitScratch* sc, int* d_status, cudaStream_t stream) {
  SplitOperand o[2];
  const int rc = split_operands(d, sc, o, stream);
  if (rc != 0) return rc;
  const int kp = o[0].kp;
  CUtensorMap ta, tb, tc;
  bool ok = d.a_mn ? make_tmap(&ta, o[0].dst, d.M, 3 * kp, o[0].pitch, 64, GEMM_BK) : make_tmap(&ta, o[0].dst, 3 * kp, d.M, o[0].pitch, GEMM_BK, 128);
  ok = ok && (d.b_mn ? make_tmap(&tb, o[1].dst, d.N, 3 * kp, o[1].pitch, 64, GEMM_BK) : make_tmap(&tb, o[1].dst, 3 * kp, d.N, o[1].pitch, GEMM_BK, 128));
  ok = ok && make_tmap(&tc, d.C, d.N, d.M, d.ldc, 32, 32, true);
  if (!ok) return -2;
  const bool accum = d.out == GEMM_OUT_ACCUM;
  const F32TcArgs a{d.M, d.N, d.K, kp, accum ? 1 : 0, parts, d.alpha, accum ? nullptr : d.res1, d.s1, accum ? nullptr : d.res2, d.s2, d.ldres,
                    reinterpret_cast<float*>(d.C), d.ldc, reinterpret_cast<const float*>(d.A), reinterpret_cast<const float*>(d.B), d.lda, d.ldb};
  const cudaError_t e = parts > 1 ? launch_f32_tc_layout<true>(d, ta, tb, tc, a, d_status, stream) : launch_f32_tc_layout<false>(d, ta, tb, tc, a, d_status, stream);
  if (e != cudaSuccess) {
    g_gemm_err = std::string("gemm_f32 tensor-core launch: ") + cudaGetErrorString(e);
    return -4;
  }
  return 0;
}

bool gemm_f32_parts(const GemmDesc& d, size_t (&bytes)[2]) {
  const int parts = d.M > 0 && d.N > 0 && d.K > 0 ? f32_on_tensor_cores(d) : 0;
  if (parts == 0) return false;
  int pitch;
  for (int i = 0; i < 2; ++i) bytes[i] = parts_bytes(d, i, &pitch);
  cudaFuncAttributes attr;
  cudaFuncGetAttributes(&attr, split_operands_kernel<3>);
  if (parts > 1) d.a_mn ? (d.b_mn ? load_f32_tc<true, true, true>() : load_f32_tc<true, false, true>())
                        : (d.b_mn ? load_f32_tc<false, true, true>() : load_f32_tc<false, false, true>());
  else d.a_mn ? (d.b_mn ? load_f32_tc<true, true, false>() : load_f32_tc<true, false, false>())
              : (d.b_mn ? load_f32_tc<false, true, false>() : load_f32_tc<false, false, false>());
  return true;
}

int gemm_f32(const GemmDesc& d, SplitScratch* sc, int* d_status, cudaStream_t stream) {
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return 0;
  if (d.out == GEMM_OUT_BF16) {
    g_gemm_err = "fp32 GEMM cannot write bf16";
    return -2;
  }
  if (const int parts = sc != nullptr ? f32_on_tensor_cores(d) : 0) {
    const int rc = gemm_f32_tc(d, parts, sc, d_status, stream);
    if (rc != GEMM_NO_SCRATCH) return rc;  // no memory for the parts: the FMA kernels need none
  }
  if (f32_aligned(d)) {
    const cudaError_t e = launch_f32(d, stream);
    if (e != cudaSuccess) {
      g_gemm_err = std::string("gemm_f32 launch: ") + cudaGetErrorString(e);
      return -4;
    }
    return 0;
  }
  dim3 grid((d.N + 63) / 64, (d.M + 63) / 64);
  gemm_f32_kernel<<<grid, 256, 0, stream>>>(
      reinterpret_cast<const float*>(d.A), reinterpret_cast<const float*>(d.B), reinterpret_cast<float*>(d.C),
      d.M, d.N, d.K, d.lda, d.ldb, d.ldc, d.a_mn ? 1 : 0, d.b_mn ? 1 : 0, d.out, d.alpha, d.res1, d.s1, d.res2,
      d.s2, d.ldres);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_gemm_err = std::string("gemm_f32 launch: ") + cudaGetErrorString(e);
    return -4;
  }
  return 0;
}

}  // namespace ane
