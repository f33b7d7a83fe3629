// The GEMM of gemm_tcgen05.cuh on CTA pairs: two CTAs of a cluster share one 256 x BN output tile and issue one
// tcgen05.mma.cta_group::2 stream.
//
// Why: a CTA that computes 128 x 256 alone reads 48 KB of operands for 512 tensor cycles, 96 bytes a cycle, and the L2
// delivers about 60 to each SM; the plain kernel therefore ran at 1.2 - 1.5 PFLOP/s whatever its epilogue. In a pair each CTA
// loads its own 128 rows of A and only HALF of the B tile (the tensor cores read the other half from the peer's shared
// memory): 32 KB for the same 512 cycles, 64 bytes a cycle, and six stages instead of four fit.
//
// Roles per CTA as in the plain kernel (TMA warp, MMA warp, epilogue warps); only rank 0 issues MMAs. `full` barriers live
// in rank 0 and count the bytes of both CTAs; commits release the stage and publish the accumulator in both CTAs; `tempty` of
// rank 0 is arrived at by the epilogue warps of both. An epilogue functor sees rows and columns exactly as in the plain kernel: the
// two warps of a lane quarter share the columns of a tile, or, where an epilogue sums over them (kWholeTiles), take tiles in turn.
#pragma once
#include "gemm_tcgen05.cuh"
#include "rope.cuh"
#include "swiglu.cuh"

namespace agrpo {

static constexpr int kPairBM = 2 * kGemmBM;

template <int BN, bool B_MN>
struct PairSmem {
  static constexpr int kABytes = kGemmBM * kGemmBK * 2;
  // an MN-major B comes in boxes of 64 columns: the half tile of BN = 192 occupies two of them
  static constexpr int kBBoxes = (BN / 2 + 63) / 64;
  static constexpr int kBBytes = (B_MN ? kBBoxes * 64 : BN / 2) * kGemmBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = kStageBytes > 28672 ? 6 : kStageBytes > 24576 ? 7 : 8;
  static constexpr int kTotal = kStages * kStageBytes + 256 + 1024;  // + barriers, alignment slack
};

__host__ __device__ inline int pair_num_items(int M, int tiles_n, int group_n) {
  const int g = group_n <= 1 ? 1 : group_n;
  return ((M + kPairBM - 1) / kPairBM) * ((tiles_n + g - 1) / g);
}

// D = acc (+ bias) (+ aux), aux being a bf16 residual (bf16 output) or what D holds already (fp32 output, the weight gradients).
// aux of a warp's next 32 columns is read while the current ones are converted; whole 32-byte sectors are read and written.
// The launcher checks that rows of D and aux start on 32 bytes and that N is a multiple of 16 (bf16) or 8 (fp32).
template <bool F32, bool AUX>
struct PairStoreEpilogue {
  void* D;
  long long ldd;
  const __nv_bfloat16* bias;  // [N] or nullptr, 16-byte aligned
  const void* aux;
  long long lda;
  int bn;              // columns a warp converts per tile
  static constexpr int kVec = F32 ? 8 : 16;
  uint32_t xn[32 / kVec][8];

  __device__ __forceinline__ void fetch(int row, int col0, int M, int N) {
    if constexpr (AUX) {
      if (row >= M) return;
#pragma unroll
      for (int i = 0; i < 32 / kVec; ++i)
        if (col0 + i * kVec < N)
          ld_global_32b(reinterpret_cast<const uint8_t*>(aux) + ((long long)row * lda + col0 + i * kVec) * (F32 ? 4 : 2), xn[i]);
    }
  }
  __device__ __forceinline__ void item_begin(int, int, int) {}
  __device__ __forceinline__ void item_end(int, int, int, int) {}
  __device__ __forceinline__ void tile_begin(int row, int col0, int M, int N) { fetch(row, col0, M, N); }
  __device__ __forceinline__ void chunk(int row, int col0, const uint32_t (&r)[32], int M, int N) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    if (bias != nullptr) {
#pragma unroll
      for (int i = 0; i < 32; i += 8)
        if (col0 + i < N) {
          const uint4 w = *reinterpret_cast<const uint4*>(bias + col0 + i);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            v[i + 2 * j] += f.x;
            v[i + 2 * j + 1] += f.y;
          }
        }
    }
    if constexpr (AUX) {
#pragma unroll
      for (int i = 0; i < 32 / kVec; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if constexpr (F32) {
            v[i * 8 + j] += __uint_as_float(xn[i][j]);
          } else {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xn[i][j]));
            v[i * 16 + 2 * j] += f.x;
            v[i * 16 + 2 * j + 1] += f.y;
          }
        }
      if (col0 % bn + 32 < bn) fetch(row, col0 + 32, M, N);
    }
    if (row >= M) return;
#pragma unroll
    for (int i = 0; i < 32 / kVec; ++i) {
      if (col0 + i * kVec >= N) break;
      uint32_t o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = F32 ? __float_as_uint(v[i * kVec + j]) : pack_bf16x2(v[i * kVec + 2 * (j & 7)], v[(i * kVec + 2 * (j & 7) + 1) & 31]);
      st_global_32b(reinterpret_cast<uint8_t*>(D) + ((long long)row * ldd + col0 + i * kVec) * (F32 ? 4 : 2), o);
    }
  }
};

// out[m, j] = silu(g) * u for a tile whose accumulator holds gate columns in its first half and up columns in its second
// (GemmShape::dual_b), g and u times the row scale of SwigluEpilogue. BF16: g and u are rounded to bf16 first, so that the
// result is bit for bit that of a plain product followed by swiglu_fwd (what fully sharded weights and short batches run); with
// gu != nullptr the two projections are stored as well ([M, 2F]: what the backward pass needs). F is a multiple of 16, rows of
// D and gu start on 32 bytes.
template <bool BF16>
struct PairSwigluEpilogue {
  static constexpr bool kDual = true;
  __nv_bfloat16* D;
  long long ldd;
  __nv_bfloat16* gu;
  long long ldgu;
  int F;
  const sumsq_t* ss_in;
  float inv_k, eps, rs;

  __device__ __forceinline__ void item_begin(int row, int M, int) {
    rs = (ss_in != nullptr && row < M) ? rsqrtf(sumsq_from_fixed(ss_in[row]) * inv_k + eps) : 1.f;
  }
  __device__ __forceinline__ void item_end(int, int, int, int) {}
  __device__ __forceinline__ void dual_chunk(int row, int col, const uint32_t (&rg)[32], const uint32_t (&ru)[32], int M) {
    if (row >= M) return;
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      if (col + c >= F) break;
      uint32_t o[8], pg[8], pu[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float2 g = make_float2(__uint_as_float(rg[c + 2 * j]), __uint_as_float(rg[c + 2 * j + 1]));
        float2 u = make_float2(__uint_as_float(ru[c + 2 * j]), __uint_as_float(ru[c + 2 * j + 1]));
        if constexpr (BF16) {
          pg[j] = pack_bf16x2(g.x, g.y);
          pu[j] = pack_bf16x2(u.x, u.y);
          g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pg[j]));
          u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pu[j]));
        } else {
          g.x *= rs; g.y *= rs; u.x *= rs; u.y *= rs;
        }
        o[j] = pack_bf16x2(g.x / (1.f + __expf(-g.x)) * u.x, g.y / (1.f + __expf(-g.y)) * u.y);
      }
      if constexpr (BF16) {
        if (gu != nullptr) {
          __nv_bfloat16* z = gu + (long long)row * ldgu + col + c;
          st_global_32b(z, pg);
          st_global_32b(z + F, pu);
        }
      }
      st_global_32b(D + (long long)row * ldd + col + c, o);
    }
  }
};

// qkv projection with bias and rotary embedding: a warp's 128 columns are one head, whose columns i and 64 + i it reads together.
// The projection is rounded to bf16 before the rotation: bit for bit a plain product followed by the rotation kernel. Heads of
// 128 columns, the first `rot_cols` columns rotate, the others (v) are stored as they are; rows of D start on 32 bytes.
struct PairRopeEpilogue {
  static constexpr bool kHalves = true;
  __nv_bfloat16* D;
  long long ldd;
  const __nv_bfloat16* bias;  // [N] or nullptr, 16-byte aligned
  AttnRope rope;
  int rot_cols;
  long long table;            // of this thread's row

  __device__ __forceinline__ void item_begin(int row, int M, int) { table = row < M ? rope.row(row) * 64 : 0; }
  __device__ __forceinline__ void item_end(int, int, int, int) {}
  // 32 columns at col and 32 at col + 64
  __device__ __forceinline__ void halves_chunk(int row, int col, const uint32_t (&ra)[32], const uint32_t (&rb)[32], int M, int N) {
    if (row >= M || col >= N) return;
    const float* ct = rope.cos_t + table + (col & 63);
    const float* st = rope.sin_t + table + (col & 63);
    const bool rotates = col < rot_cols;
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      uint32_t oa[8], ob[8];
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        float a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a[k] = __uint_as_float(ra[c + j + k]);
          b[k] = __uint_as_float(rb[c + j + k]);
        }
        if (bias != nullptr) {
          const uint2 wa = *reinterpret_cast<const uint2*>(bias + col + c + j), wb = *reinterpret_cast<const uint2*>(bias + col + 64 + c + j);
          const float2 a0 = unpack(wa.x), a1 = unpack(wa.y), b0 = unpack(wb.x), b1 = unpack(wb.y);
          a[0] += a0.x; a[1] += a0.y; a[2] += a1.x; a[3] += a1.y;
          b[0] += b0.x; b[1] += b0.y; b[2] += b1.x; b[3] += b1.y;
        }
        if (rotates) {
          const float4 cs = *reinterpret_cast<const float4*>(ct + c + j), sn = *reinterpret_cast<const float4*>(st + c + j);
          const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            a[k] = __bfloat162float(__float2bfloat16(a[k]));
            b[k] = __bfloat162float(__float2bfloat16(b[k]));
            rope_rotate(a[k], b[k], cv[k], sv[k]);
          }
        }
        oa[j / 2] = pack_bf16x2(a[0], a[1]);
        oa[j / 2 + 1] = pack_bf16x2(a[2], a[3]);
        ob[j / 2] = pack_bf16x2(b[0], b[1]);
        ob[j / 2 + 1] = pack_bf16x2(b[2], b[3]);
      }
      __nv_bfloat16* d = D + (long long)row * ldd + col + c;
      st_global_32b(d, oa);
      st_global_32b(d + 64, ob);
    }
  }
  __device__ __forceinline__ static float2 unpack(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
};

// Input gradient of the down projection taken on to the gate / up projections: D[m, j] and D[m, F + j] are the gradients of g and u
// where the product is that of silu(g) * u. The product is rounded to bf16 first: bit for bit a plain product followed by
// swiglu_bwd. g and u of a warp's next 32 columns are read while the current ones are converted. F is a multiple of 16, rows of
// gu and D start on 32 bytes.
struct PairSwigluBwdEpilogue {
  __nv_bfloat16* D;         // [M, 2F]
  long long ldd;
  const __nv_bfloat16* gu;  // [M, 2F]
  long long ldgu;
  int F;
  int bn;                   // columns a warp converts per tile
  uint32_t g[2][8], u[2][8];

  __device__ __forceinline__ void fetch(int row, int col0, int M) {
    if (row >= M) return;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (col0 + i * 16 < F) {
        const __nv_bfloat16* p = gu + (long long)row * ldgu + col0 + i * 16;
        ld_global_32b(p, g[i]);
        ld_global_32b(p + F, u[i]);
      }
  }
  __device__ __forceinline__ void item_begin(int, int, int) {}
  __device__ __forceinline__ void item_end(int, int, int, int) {}
  __device__ __forceinline__ void tile_begin(int row, int col0, int M, int) { fetch(row, col0, M); }
  __device__ __forceinline__ void chunk(int row, int col0, const uint32_t (&r)[32], int M, int N) {
    uint32_t dg[2][8], du[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t d2 = pack_bf16x2(__uint_as_float(r[i * 16 + 2 * j]), __uint_as_float(r[i * 16 + 2 * j + 1]));
        const float2 gf = unpack(g[i][j]), uf = unpack(u[i][j]), df = unpack(d2);
        float2 a, b;
        swiglu_grad(gf.x, uf.x, df.x, a.x, b.x);
        swiglu_grad(gf.y, uf.y, df.y, a.y, b.y);
        dg[i][j] = pack_bf16x2(a.x, a.y);
        du[i][j] = pack_bf16x2(b.x, b.y);
      }
    if (col0 % bn + 32 < bn) fetch(row, col0 + 32, M);
    if (row >= M) return;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (col0 + i * 16 < N) {
        __nv_bfloat16* d = D + (long long)row * ldd + col0 + i * 16;
        st_global_32b(d, dg[i]);
        st_global_32b(d + F, du[i]);
      }
  }
  __device__ __forceinline__ static float2 unpack(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
};

template <class Epi, class = void>
struct EpiHalves { static constexpr bool value = false; };
template <class Epi>
struct EpiHalves<Epi, decltype((void)Epi::kHalves)> { static constexpr bool value = Epi::kHalves; };

template <class Epi, class = void>
struct EpiWholeTiles { static constexpr bool value = false; };
template <class Epi>
struct EpiWholeTiles<Epi, decltype((void)Epi::kWholeTiles)> { static constexpr bool value = Epi::kWholeTiles; };

template <class Epi, class = void>
struct EpiDual { static constexpr bool value = false; };
template <class Epi>
struct EpiDual<Epi, decltype((void)Epi::kDual)> { static constexpr bool value = Epi::kDual; };

// Which tile width a plain product takes. A pair needs about 1 : 0.80 : 0.60 of the time of a 256-wide tile for 192 and 128
// columns (measured at 31287 x 1536 x 8960: 546, 591, 638 us; a 192-wide MN-major tile of B is loaded as 256 columns and takes
// 0.86), so a narrower tile pays where it saves a wave: at 6223 x 1536 x 8960 the 150 tiles of 256 columns need 3 waves of 74
// pairs (153 us), 200 tiles of 192 columns need 3 cheaper ones (124 us); 1536 x 1536 x 31287 is 36 tiles (218 us) or 72 (130 us).
// A width is a multiple of `unit`.
inline int pair_pick_bn(int M, int N, bool b_mn, int num_sms, int n1 = 0, int unit = 1) {
  const int pairs = num_sms / 2 > 0 ? num_sms / 2 : 1;
  const int cands[3] = {256, 192, 128};
  const float cost[3] = {1.f, b_mn ? 0.86f : 0.80f, 0.60f};
  int best = 256;
  float best_t = 0.f;
  for (int i = 0; i < 3; ++i) {
    const int bn = cands[i];
    if (bn % unit != 0) continue;
    const int tiles_n = n1 > 0 ? (n1 + bn - 1) / bn + (N - n1 + bn - 1) / bn : (N + bn - 1) / bn;
    const int items = pair_num_items(M, tiles_n, 1);
    const float t = (float)((items + pairs - 1) / pairs) * cost[i];
    if (i == 0 || t < best_t) {
      best = bn;
      best_t = t;
    }
  }
  return best;
}
// One 128-row tile cannot feed a pair.
inline bool pair_serves(int M, int num_sms) { return M > kGemmBM && num_sms >= 2; }

// Work-item order: bands of 8 row tiles, row fastest, then columns (or groups of columns), so that the pairs that run at the
// same time share A and B through L2 whatever K is: 74 pairs hold 8 x 256 rows of A and about 9 column tiles of B.
__device__ __forceinline__ void pair_item_coords(int idx, int tiles_m, int tiles_n, int group_n, int& tm, int& tn0, int& count) {
  constexpr int kBand = 8;
  const int g = group_n <= 1 ? 1 : group_n;
  const int groups = (tiles_n + g - 1) / g;
  const int band = idx / (kBand * groups);
  const int rem = idx - band * kBand * groups;
  const int rows = min(kBand, tiles_m - band * kBand);
  tm = band * kBand + rem % rows;
  tn0 = (rem / rows) * g;
  count = min(g, tiles_n - tn0);
}

template <int BN, bool A_MN, bool B_MN, class Epi, int EW>
__global__ void __launch_bounds__(64 + EW * 32, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmShape p, Epi epi) {
  using S = PairSmem<BN, B_MN>;
  constexpr int kStages = S::kStages;
  constexpr uint32_t kTmemCols = BN > 128 ? 512 : 256;
  constexpr int kTmemBuf = kTmemCols / 2;  // columns from one accumulator to the other
  constexpr bool kWhole = EpiWholeTiles<Epi>::value;
  static_assert(!kWhole || EW == 8, "two warps per lane quarter, one per accumulator");
  constexpr int kEpiCols = kWhole ? BN : BN / (EW / 4);  // columns of a tile that one epilogue warp converts
  constexpr uint32_t kIdesc = umma_idesc_bf16(kPairBM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * S::kStageBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tfull_bar = empty_bar + kStages;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int tiles_m = (p.M + kPairBM - 1) / kPairBM;
  const int tiles_n = p.tiles_n(BN);
  const int num_items = pair_num_items(p.M, tiles_n, p.group_n);
  const int num_kb = (p.K + kGemmBK - 1) / kGemmBK;
  const int my_pair = (int)blockIdx.x >> 1;
  const int stride = (int)gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);   // rank 0's own arrival; the bytes of both CTAs complete it
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], kWhole ? EW : 2 * EW);  // the epilogue warps of both CTAs
    }
    fence_mbar_init();
    fence_cluster_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers and tensor memory are ready
  tc_fence_after();
  pdl_wait();
  pdl_launch();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = my_pair; item < num_items && ok; item += stride) {
        int tm, tn0, count;
        pair_item_coords(item, tiles_m, tiles_n, p.group_n, tm, tn0, count);
        const int m0 = tm * kPairBM + rank * kGemmBM;
        for (int t = 0; t < count && ok; ++t) {
          const int n0 = p.first_col(tn0 + t, BN);
          const int a0 = p.second(tn0 + t, BN) ? p.a2 : 0;
          // two products side by side in one tile: rank 0 holds the gate rows of B, rank 1 the up rows
          const int b0 = p.dual_b > 0 ? n0 / 2 + rank * p.dual_b : n0 + rank * (BN / 2);
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
              report_status(p.status, kStatusWaitEmptyTimeout);
              ok = false;
              break;
            }
            uint8_t* sa = smem + stage * S::kStageBytes;
            uint8_t* sb = sa + S::kABytes;
            if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * S::kStageBytes);
            const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0);
            const int k0 = kb * kGemmBK;
            if constexpr (!A_MN) {
              tma_load_2d_pair(sa, &tmA, bar, a0 + k0, m0);
            } else {
#pragma unroll
              for (int j = 0; j < kGemmBM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmA, bar, m0 + j * 64, k0);
            }
            if constexpr (!B_MN) {
              tma_load_2d_pair(sb, &tmB, bar, k0, b0);
            } else {
#pragma unroll
              for (int j = 0; j < S::kBBoxes; ++j) tma_load_2d_pair(sb + j * 8192, &tmB, bar, b0 + j * 64, k0);
            }
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (rank 0) ------------------------------
    if (rank == 0 && elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      bool ok = true;
      for (int item = my_pair; item < num_items && ok; item += stride) {
        int tm, tn0, count;
        pair_item_coords(item, tiles_m, tiles_n, p.group_n, tm, tn0, count);
        for (int t = 0; t < count && ok; ++t, ++local) {
          const int buf = local & 1;
          if (!mbar_wait_cluster(&tempty_bar[buf], ((local >> 1) & 1) ^ 1)) {
            report_status(p.status, kStatusWaitTmemEmptyTimeout);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + buf * kTmemBuf;
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!mbar_wait_cluster(&full_bar[stage], phase)) {
              report_status(p.status, kStatusWaitFullTimeout);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * S::kStageBytes);
            const uint32_t sb = sa + S::kABytes;
#pragma unroll
            for (int k = 0; k < kGemmBK / 16; ++k) {
              const uint64_t da = A_MN ? umma_smem_desc(sa + k * 2048, 8192, 1024) : umma_smem_desc(sa + k * 32, 16, 1024);
              const uint64_t db = B_MN ? umma_smem_desc(sb + k * 2048, 8192, 1024) : umma_smem_desc(sb + k * 32, 16, 1024);
              tc_mma_f16_pair(tmem_d, da, db, kIdesc, (kb > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit_pair(&empty_bar[stage]);
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (ok) tc_commit_pair(&tfull_bar[buf]);
        }
      }
    }
  } else {
    // ------------------------------ Epilogue ------------------------------
    const int quarter = warp & 3;
    const int turn = (warp - 2) >> 2;
    const int part = kWhole ? 0 : turn;  // which kEpiCols columns of a tile
    int local = 0;
    bool ok = true;
    for (int item = my_pair; item < num_items && ok; item += stride) {
      int tm, tn0, count;
      pair_item_coords(item, tiles_m, tiles_n, p.group_n, tm, tn0, count);
      if constexpr (kWhole) {  // an item is one tile
        if ((local & 1) != turn) {
          ++local;
          continue;
        }
      }
      const int row = tm * kPairBM + rank * kGemmBM + quarter * 32 + lane;
      epi.item_begin(row, p.M, p.N);
      for (int t = 0; t < count; ++t, ++local) {
        const int buf = local & 1;
        const int n0 = p.first_col(tn0 + t, BN) + part * kEpiCols, n_end = p.end_col(tn0 + t, BN);
        epi_tile_begin(epi, row, n0, p.M, n_end, 0);
        if (!mbar_wait(&tfull_bar[buf], (local >> 1) & 1)) {
          report_status(p.status, kStatusWaitTmemFullTimeout);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * kTmemBuf + part * kEpiCols;
        if constexpr (EpiDual<Epi>::value) {
          // the warps of a quarter share the tile's BN / 2 output columns
          const uint32_t gate = taddr - part * (kEpiCols / 2);
          const int col = (tn0 + t) * (BN / 2) + part * (kEpiCols / 2);
#pragma unroll 1
          for (int c = 0; c < kEpiCols / 64; ++c) {
            uint32_t g[32], u[32];
            tmem_ld_32x32(gate + c * 32, g);
            tmem_ld_32x32(gate + BN / 2 + c * 32, u);
            tc_wait_ld();
            epi.dual_chunk(row, col + c * 32, g, u, p.M);
          }
        } else if constexpr (EpiHalves<Epi>::value) {
          static_assert(kEpiCols == 128, "a warp's columns are one head");
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            uint32_t a[32], b[32];
            tmem_ld_32x32(taddr + c * 32, a);
            tmem_ld_32x32(taddr + 64 + c * 32, b);
            tc_wait_ld();
            epi.halves_chunk(row, n0 + c * 32, a, b, p.M, n_end);
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < kEpiCols / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c * 32, r);
            tc_wait_ld();
            epi.chunk(row, n0 + c * 32, r, p.M, n_end);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&tempty_bar[buf]), 0));
      }
      if (ok) epi.item_end(row, p.M, p.N, (p.group_n <= 1 ? tn0 : tn0 / p.group_n) * (EW / 4) + part);
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer may still read this CTA's operands or arrive at its barriers until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// Tensor maps must have boxes of 64 x 128 for a K-major A, 64 x (BN / 2) for a K-major B, 64 x 64 for MN-major operands.
template <int BN, bool A_MN, bool B_MN, int EW = 8, class Epi>
inline void gemm_pair_launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmShape& p, const Epi& epi, int num_sms,
                             cudaStream_t stream) {
  using S = PairSmem<BN, B_MN>;
  auto kernel = gemm_pair_kernel<BN, A_MN, B_MN, Epi, EW>;
  AGRPO_SET_MAX_DYN_SMEM(kernel, S::kTotal, "gemm pair smem attr");
  const int items = pair_num_items(p.M, p.tiles_n(BN), p.group_n);
  const int pairs = num_sms / 2 > 0 ? num_sms / 2 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (items < pairs ? items : pairs));
  cfg.blockDim = dim3(64 + EW * 32);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_flag() ? 2 : 1;
  check_cuda(cudaLaunchKernelEx(&cfg, kernel, ta, tb, p, epi), "gemm_pair launch");
}

}  // namespace agrpo
