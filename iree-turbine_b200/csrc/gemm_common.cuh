// Pieces shared by the GEMM kernels (the persistent whole-tile kernel and the split-K cluster
// kernel): tile constants, the kernel parameter block, the shared-memory layout of the operand
// ring, tile rasterisation and the epilogue helpers.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace b200k {
namespace gemm_detail {

constexpr int kBM = 128;
constexpr int kBKBytes = 128;
constexpr int kGemmThreads = 192;
constexpr int kGroupRows = 2048;  // rows of a rasterisation group (keeps one wave's operands L2-resident)

enum GemmKind : int { kKindF16 = 0, kKindBF16 = 1, kKindE4M3 = 2 };

struct GemmParams {
  void* c;
  const float* scale_a;
  const float* scale_b;
  int32_t* status;
  int64_t ldc;
  int32_t m, n;
  int32_t tiles_m, tiles_n, num_kb;  // tiles_m counts tiles of 128 rows, or 256 of a pair, num_kb pipeline stages along K
  int32_t stage_bytes;               // bytes the loads of a pipeline stage bring, of both CTAs of a pair
  int32_t batch;                     // independent problems (tensor maps are 3-D: [batch][rows][k])
  int32_t split;                     // split-K kernel only: CTAs per tile (= cluster size) ...
  int32_t kb_per_split;              // ... each summing this many consecutive stages
  int64_t c_batch_stride;            // elements between the C matrices of consecutive problems
  // Optional fused epilogue: y = act(acc * scale + bias[col]); bias == nullptr and act == 0 leave
  // the plain path untouched.
  const void* bias;
  int32_t bias_dtype;  // B200K_F32 | B200K_F16 | B200K_BF16
  int32_t act;         // B200K_ACT_*
  // Operand storage (generic kernel only): a_mn = A is stored [K, M] (M contiguous), b_mn = B is
  // stored [K, N] (N contiguous); 0 = the contraction dimension K is the contiguous one.
  int32_t a_mn, b_mn;
  // MN-major and a multiple of 64 long: the tensor map is 4-D ([batch][R / 64][K][64]) and one load brings all
  // 64-element blocks of a stage; else one 3-D load per block, which clips at R.
  int32_t a_blocks, b_blocks;
  int32_t vec_store_ok;
  int32_t tma_store_ok;  // C's base, row pitch and row length are multiples of 16 bytes: epilogue uses TMA stores
  int32_t store_bytes;   // otherwise: widest store (2, 4 or 8 bytes) that C's base and pitches allow
  // Fused all-gather of a column shard: when num_peers > 0 every output tile is written with plain
  // 16-byte stores into each peer's full matrix (peer-mapped memory) at column peer_col0.
  int32_t num_peers;
  int32_t peer_first;  // index of the first peer written (the rank after this one); own copy last
  int64_t peer_ldc;
  int64_t peer_col0;
  void* peers[8];
  void* peer_mc;  // NVSwitch multicast address of the matrix, or nullptr
  int32_t peer_tma;  // the pieces go out as bulk tensor stores through PeerMaps (one per rank)
};

// Tensor maps over this rank's column shard inside every rank's full matrix (fused all-gather):
// map i covers columns [col0, col0 + n) of rank i's matrix, so a store is clipped at the shard's edge.
struct PeerMaps {
  CUtensorMap m[8];
};

template <int BN, int CTAS>
struct GemmSmem {
  // k-blocks (128 bytes of K) per pipeline stage.  The thread that issues the MMAs spends about 50 cycles
  // on each of a block's four and 280 more per stage on the barrier wait, the commit and the loop (measured
  // with that thread behind lane == 0; behind elect.sync an MMA of N = 64 takes it 49 cycles, see elect_one).  For a
  // tile whose MMAs execute in 64 cycles or less that thread, not the tensor core or the loads, set the
  // pace (480 cycles per block, for BN = 64 as for BN = 128), so those tiles take two blocks per stage.
  static constexpr int kSub = BN <= 128 ? 2 : 1;
  static constexpr int kStages = CTAS == 2 ? 6 : (BN == 128 ? 3 : 4);
  static constexpr int kABytes = kBM * kBKBytes;  // per k-block; a CTA of a pair holds its rows of A and its half of B
  static constexpr int kBBytes = BN / CTAS * kBKBytes;
  static constexpr int kBOffset = kSub * kABytes;  // a stage: A blocks, then B blocks
  static constexpr int kStageBytes = kSub * (kABytes + kBBytes);
  // epilogue staging: eight 32-row x 128-byte buffers (TMA store source)
  static constexpr int kStagingOffset = kStages * kStageBytes;
  static constexpr int kStagingBytes = 8 * 32 * 128;
  static constexpr int kBarOffset = kStagingOffset + kStagingBytes;
  static constexpr int kNumBars = 2 * kStages + 4;
  static constexpr int kBiasOffset = kBarOffset + kNumBars * 8 + 16;  // the tile's bias as fp32
  static_assert(kBiasOffset % 16 == 0, "bias is read as float4");
  static constexpr int kTotal = kBiasOffset + BN * 4;
  static constexpr int kDynamic = kTotal + 1024;  // slack for 1024-byte alignment of the tiles
};

template <int ROWS>  // of a tile
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
  constexpr int kGroupM = kGroupRows / ROWS;
  const int group_size = kGroupM * tiles_n;
  const int group = t / group_size;
  const int first_m = group * kGroupM;
  const int gm = min(tiles_m - first_m, kGroupM);
  const int r = t - group * group_size;
  tm = first_m + r % gm;
  tn = r / gm;
}

// One box of a k-block of an operand.  CTAS == 2: counted on the barrier of the pair's leader.
template <int CTAS>
__device__ __forceinline__ void load_3d(uint8_t* dst, const CUtensorMap* tmap, uint64_t* bar, int c0, int c1, int c2) {
  if constexpr (CTAS == 2)
    tma_load_3d_pair(dst, tmap, cluster_map_shared(smem_u32(bar), 0), c0, c1, c2);
  else
    tma_load_3d(dst, tmap, bar, c0, c1, c2);
}

// One k-block of an MN-major operand: R rows or columns of the tile (64-element blocks 8 KB apart), 64 K-rows.
template <int R, int CTAS = 1>
__device__ __forceinline__ void load_mn_major(uint8_t* dst, const CUtensorMap* tmap, uint64_t* bar, int r0, int k0, int bz,
                                              bool blocks) {
  if (blocks) {
    if constexpr (CTAS == 2)
      tma_load_4d_pair(dst, tmap, cluster_map_shared(smem_u32(bar), 0), 0, k0, r0 >> 6, bz);
    else
      tma_load_4d(dst, tmap, bar, 0, k0, r0 >> 6, bz);
  } else {
#pragma unroll
    for (int b = 0; b < R / 64; ++b) load_3d<CTAS>(dst + b * 8192, tmap, bar, r0 + b * 64, k0, bz);
  }
}

template <typename OutT>
__device__ __forceinline__ OutT to_out(float v);
template <>
__device__ __forceinline__ float to_out<float>(float v) {
  return v;
}
template <>
__device__ __forceinline__ __half to_out<__half>(float v) {
  return __float2half_rn(v);
}
template <>
__device__ __forceinline__ __nv_bfloat16 to_out<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

template <int ACT>
__device__ __forceinline__ float apply_act(float x) {
  if constexpr (ACT == B200K_ACT_RELU) return fmaxf(x, 0.f);
  if constexpr (ACT == B200K_ACT_GELU)  // exact (erf) form, the default of aten::gelu
    return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
  if constexpr (ACT == B200K_ACT_SILU) {
    // x / (1 + e^-x): quotient by a hardware reciprocal, corrected by its own residual (Markstein 1990).  Over
    // 524288 values of -95 to 95 not a bit differs from the IEEE division, which branches to a slow path per
    // element (8000 x 1024 x 1024: 147 us with it, 26.6 now, 21.2 without an activation; 24.0 with the reciprocal
    // alone refined, whose results were up to one unit further off).  Numerator and denominator are divided
    // by 16, which keeps the reciprocal of the largest 1 + e^-x a normal number.  Where the residual is NaN
    // (1 + e^-x or x infinite) the uncorrected quotient is the answer: a zero below -88.7, x at +infinity,
    // NaN at -infinity.
    const float d = fmaf(__expf(-x), 0.0625f, 0.0625f), num = x * 0.0625f;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = num * r, residual = fmaf(-d, q, num);
    return residual == residual ? fmaf(residual, r, q) : q;
  }
  return x;
}

__device__ __forceinline__ float apply_act(float x, int act) {
  switch (act) {
    case B200K_ACT_RELU:
      return apply_act<B200K_ACT_RELU>(x);
    case B200K_ACT_GELU:
      return apply_act<B200K_ACT_GELU>(x);
    case B200K_ACT_SILU:
      return apply_act<B200K_ACT_SILU>(x);
    default:
      return x;
  }
}

__device__ __forceinline__ float load_bias(const void* bias, int dtype, int col) {
  if (dtype == B200K_F32) return reinterpret_cast<const float*>(bias)[col];
  if (dtype == B200K_F16) return __half2float(reinterpret_cast<const __half*>(bias)[col]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[col]);
}

// acc * scale + bias, then the activation, on N accumulator values of one row, in place.  `bias` is the
// fp32 bias of these columns in shared memory (16-byte aligned, the same for every lane, so a float4
// read is a broadcast); afterwards the caller's own scaling must be 1.  The activation is chosen
// outside the loop: with the choice (and a bias load that picked its data type) inside, the 64-fold
// unrolled body made a 3000 x 4352 x 3840 product with bias take 155 us instead of 118.
template <int N>
__device__ __forceinline__ void fused_epilogue(uint32_t (&r)[N], float scale, const float* bias, int act) {
#pragma unroll
  for (int j = 0; j < N; j += 4) {
    const float4 b = *reinterpret_cast<const float4*>(bias + j);
    r[j] = __float_as_uint(__uint_as_float(r[j]) * scale + b.x);
    r[j + 1] = __float_as_uint(__uint_as_float(r[j + 1]) * scale + b.y);
    r[j + 2] = __float_as_uint(__uint_as_float(r[j + 2]) * scale + b.z);
    r[j + 3] = __float_as_uint(__uint_as_float(r[j + 3]) * scale + b.w);
  }
  if (act == B200K_ACT_RELU) {
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __float_as_uint(apply_act<B200K_ACT_RELU>(__uint_as_float(r[j])));
  } else if (act == B200K_ACT_GELU) {
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __float_as_uint(apply_act<B200K_ACT_GELU>(__uint_as_float(r[j])));
  } else if (act == B200K_ACT_SILU) {
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __float_as_uint(apply_act<B200K_ACT_SILU>(__uint_as_float(r[j])));
  }
}

// One 128-byte piece of a row of C out of N = 128 / sizeof(OutT) accumulator values, as eight 16-byte chunks.
template <typename OutT, int N>
__device__ __forceinline__ void pack_row(const uint32_t (&r)[N], float scale, uint4 (&v)[8]) {
  static_assert(N * sizeof(OutT) == 128, "a piece is 128 bytes");
  constexpr int kPer = 16 / static_cast<int>(sizeof(OutT));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    union {
      uint4 u;
      OutT e[kPer];
    } pk;
#pragma unroll
    for (int j = 0; j < kPer; ++j) pk.e[j] = to_out<OutT>(__uint_as_float(r[kPer * i + j]) * scale);
    v[i] = pk.u;
  }
}

// Writes a staged piece (32 rows x 128 bytes, 16-byte chunks XOR-swizzled by row) to a matrix whose
// rows are not 16-byte aligned, V bytes per lane: lanes side by side write neighbouring bytes, so an
// instruction covers whole sectors of 1 (V = 4), 2 (V = 8) rows or half of one (V = 2).  (One row
// per lane instead, a column per instruction, touched 32 sectors each time: a 6388 x 1446 x 1440 fp8
// product took 129 us that way.)
template <typename OutT, typename V>
__device__ __forceinline__ void store_piece(OutT* c, int64_t ldc, const uint8_t* buf, int lane, int rows, int cols) {
  constexpr int kPerRow = 128 / static_cast<int>(sizeof(V));
  constexpr int kElems = static_cast<int>(sizeof(V) / sizeof(OutT));
#pragma unroll 4
  for (int u = lane; u < 32 * kPerRow; u += 32) {
    const int lr = u / kPerRow;
    const int byte = (u % kPerRow) * static_cast<int>(sizeof(V));
    const V val = *reinterpret_cast<const V*>(buf + lr * 128 + (((byte >> 4) ^ (lr & 7)) << 4) + (byte & 15));
    const int col = byte / static_cast<int>(sizeof(OutT));
    OutT* dst = c + static_cast<int64_t>(lr) * ldc + col;
    if (lr < rows) {
      // a row pitch that allows V-byte stores may still end inside one (C is a column slice)
      if (col + kElems <= cols) {
        *reinterpret_cast<V*>(dst) = val;
      } else {
        union {
          V v;
          OutT e[kElems];
        } pk;
        pk.v = val;
#pragma unroll
        for (int i = 0; i < kElems; ++i)
          if (col + i < cols) dst[i] = pk.e[i];
      }
    }
  }
}

template <typename OutT>
__device__ __forceinline__ void store_piece_any(OutT* c, int64_t ldc, const uint8_t* buf, int lane, int rows, int cols,
                                                int store_bytes) {
  if (store_bytes == 8)
    store_piece<OutT, uint2>(c, ldc, buf, lane, rows, cols);
  else if (sizeof(OutT) == 4 || store_bytes == 4)
    store_piece<OutT, uint32_t>(c, ldc, buf, lane, rows, cols);
  else if constexpr (sizeof(OutT) == 2)
    store_piece<OutT, uint16_t>(c, ldc, buf, lane, rows, cols);
}

}  // namespace gemm_detail

// Split-K kernel (gemm_splitk_sm100.cu).  Tensor maps as for the whole-tile kernel with 128-row A
// boxes; p.split in {2, 4, 8}, grid = tiles * p.split.
int launch_gemm_splitk(const CUtensorMap& ta, const CUtensorMap& tb, const gemm_detail::GemmParams& p, int bn,
                       int in_dtype, int out_dtype, cudaStream_t stream);
// Clusters of `split` CTAs of that kernel the current device holds at once (0 = cannot launch).
int splitk_resident_clusters(int bn, int split);

}  // namespace b200k
