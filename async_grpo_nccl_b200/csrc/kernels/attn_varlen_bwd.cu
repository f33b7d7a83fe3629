// Causal varlen flash-attention backward with native GQA on tcgen05.
//
// The reference gets this pass from flash-attn's autograd function behind flash_attn_varlen_func
// (gpu_process_worker.py:265-276), on K/V that were first repeated to the query head count.
//
// One CTA owns one 128-key tile of one kv head and walks over the query heads of its group and the
// query tiles at or below the diagonal. Per step five tcgen05 GEMMs run with every accumulator in
// tensor memory (512 columns: R1 = S^T then P^T, R2 = dP^T then dQ, dV, dK):
//   S^T  = K Q^T          dP^T = V dO^T                 (operands from shared memory, TMA-fed)
//   dV  += P^T dO                                       (P^T read back from tensor memory)
//   dQ   = dS K           dK  += dS^T Q                 (one dS^T tile in shared memory, read MN-major and K-major)
// dK / dV leave as bf16 once per CTA; dQ partial tiles are added to an fp32 accumulator by TMA from a buffer of their own
// (whole lines; as 16-byte reductions of single threads, 4096 a step, they were what
// a step waited for) and converted by attn_bwd_finalize_kernel. Where rotary embedding came before the attention,
// both take its transpose along on the way out.
//
// Where one CTA per (key tile, kv head) would leave SMs idle or waiting for the longest one, the group's
// query heads are dealt to several CTAs. Each stores its fp32 dK / dV, and a second kernel adds them up in order: unlike dQ, whose
// tiles arrive in any order, dK and dV repeat bit for bit. Only rows of the tiles are written.
//
// A step is a chain (S and dP, then the softmax gradient, then three products, then the read-out of dQ), and neither the 512
// columns nor the 227 KB leave room for a second tile. So the two halves of a step are kept apart and its links run beside each
// other. The tensor core goes dV(i), S(i+1), dQ(i), dK(i), dP(i+1); dS^T lives in shared memory alone, so R1 is
// free for S(i+1) as soon as dV(i) is issued, and the exponentials of a step need only S, its gradient only dP. R2 is handed back once
// dQ is in registers; half of it leaves at once, the other half behind the next step's exponentials, and no step waits for the
// reduction before the buffer is needed again. Row statistics are loaded a step ahead. Eight warps share the elementwise part,
// two per lane quarter with 64 queries each; P^T of a warp stays inside the columns that it read S^T from (queries 64.. at column 64).
//
// Measured (12 query, 2 kv heads, head_dim 128), before with one chain per step, then as it is: 31287 tokens in 11 sequences
// 2349 -> 1581 us (714 TFLOP/s), 8 x 4096 2064 -> 1335, 19 x 330 142 -> 125, 1 x 759 69 -> 55; 28 query, 4 kv heads, 25415 tokens
// 2553 -> 1729. Bound by the elementwise warps between the products: staging dQ for its reduction is 17 % of a step,
// the exponentials are a small part.
#include <cuda_bf16.h>

#include "../common/f32x2.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "../launchers.h"
#include "rope.cuh"

namespace agrpo {

namespace {

constexpr int kT = 128;  // tile edge (keys per CTA, queries per step)
constexpr int kBwdThreads = 320;

struct AttnBwdParams {
  const int4* tiles;  // {seq_start, seq_len, k0, unused}
  const float* lse;   // [Hq, T]
  const float* delta; // [Hq, T]
  __nv_bfloat16* dk;  // row pitch ldk, head h at column dk_col0 + h*D
  __nv_bfloat16* dv;
  long long ld_dk, ld_dv;
  int dk_col0, dv_col0;
  int T, Hq, Hkv, group;
  int pieces;         // CTAs that share the query heads of a (key tile, kv head)
  float* dkv;         // pieces > 1: dK / dV go here (part_offset)
  int q_col0, k_col0, v_col0;
  float scale, scale_log2;
  AttnRope rope;      // transposed rotation of dK, off when pos == nullptr
  int* status;
};

__device__ __forceinline__ void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Where the 32 rows `quarter` of a tile and head (K's heads, then V's) of one piece start: [D / 4 column groups][32 rows][4 columns],
// the order in which a warp reads them from tensor memory.
template <int D>
__device__ __forceinline__ long long part_offset(int piece, int n_tiles, int tile, int Hkv, int head, int quarter) {
  return ((((long long)piece * n_tiles + tile) * 2 * Hkv + head) * 4 + quarter) * (32 * D);
}

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmDQ, const AttnBwdParams p) {
  constexpr int kChunks = D / 64;
  constexpr int kTileBytes = kT * D * 2;
  constexpr int kChunkBytes = kT * 128;     // one 64-column swizzle chunk of a 128-row tile
  constexpr int kDsBytes = kT * kT * 2;
  constexpr int kOutBytes = 8 * 4096;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kIdescST = umma_idesc_bf16(kT, kT, 0, 0);  // S^T, dP^T: both operands K-major
  constexpr uint32_t kIdescKV = umma_idesc_bf16(kT, D, 0, 1);   // dV, dK: A from TMEM, B MN-major
  constexpr uint32_t kIdescDQ = umma_idesc_bf16(kT, D, 1, 1);   // dQ: A (dS^T in smem) MN-major, B MN-major

  // no slack to align by hand: the tiles, the buffer of dQ and the row statistics fill what a block may have
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023) != 0) {
    if (threadIdx.x == 0) report_status(p.status, kStatusBadIndex);
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sV = sK + kTileBytes;
  uint8_t* sQ = sV + kTileBytes;           // two stages
  uint8_t* sDO = sQ + 2 * kTileBytes;
  uint8_t* sDS = sDO + kTileBytes;
  uint8_t* sOut = sDS + kDsBytes;           // dQ on its way out
  float* sLse = reinterpret_cast<float*>(sOut + kOutBytes);  // [2][128], minus the log-sum
  float* sDelta = sLse + 2 * kT;                           // [2][128], minus the row product
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDelta + 2 * kT);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;   // [2]
  uint64_t* q_empty = bars + 3;  // [2]
  uint64_t* do_full = bars + 5;
  uint64_t* s_full = bars + 6;
  uint64_t* dp_full = bars + 7;
  uint64_t* p_ready = bars + 8;
  uint64_t* ds_ready = bars + 9;
  uint64_t* dv_done = bars + 10;
  uint64_t* dq_full = bars + 11;
  uint64_t* dq_read = bars + 12;
  uint64_t* all_done = bars + 13;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_head = blockIdx.x / p.pieces, piece = blockIdx.x - kv_head * p.pieces;
  const int head0 = kv_head * p.group + piece * p.group / p.pieces;  // first of this CTA's query heads
  // The table is sorted for the forward pass (heaviest query tile first); the heaviest key tile is the last.
  const int tile_idx = gridDim.y - 1 - blockIdx.y;
  const int4 tile = p.tiles[tile_idx];
  const int seq_start = tile.x, seq_len = tile.y, k0 = tile.z;
  const int n_q = (seq_len - k0 + kT - 1) / kT;
  const int n_it = n_q * ((piece + 1) * p.group / p.pieces - piece * p.group / p.pieces);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(&q_full[0], 1);
    mbar_init(&q_full[1], 1);
    mbar_init(&q_empty[0], 1);
    mbar_init(&q_empty[1], 1);
    mbar_init(do_full, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(all_done, 1);
    mbar_init(dv_done, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, 8);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_launch();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_R1 = tmem_base;        // S^T -> P^T (bf16)
  const uint32_t tmem_R2 = tmem_base + 128;  // dP^T -> dQ
  const uint32_t tmem_dV = tmem_base + 256;
  const uint32_t tmem_dK = tmem_base + 256 + D;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * kTileBytes);
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        tma_load_2d(sK + c * kChunkBytes, &tmK, kv_full, p.k_col0 + kv_head * D + c * 64, seq_start + k0);
        tma_load_2d(sV + c * kChunkBytes, &tmV, kv_full, p.v_col0 + kv_head * D + c * 64, seq_start + k0);
      }
      for (int it = 0; it < n_it; ++it) {
        const int hg = it / n_q, qt = it - hg * n_q;
        const int head = head0 + hg;
        const int row = seq_start + k0 + qt * kT;
        const int s = it & 1;
        if (it >= 2 && !mbar_wait(&q_empty[s], ((it >> 1) - 1) & 1)) {
          report_status(p.status, kStatusWaitEmptyTimeout);
          break;
        }
        mbar_expect_tx(&q_full[s], kTileBytes);
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
          tma_load_2d(sQ + s * kTileBytes + c * kChunkBytes, &tmQ, &q_full[s], p.q_col0 + head * D + c * 64, row);
        if (it >= 1 && !mbar_wait(dv_done, (it - 1) & 1)) {
          report_status(p.status, kStatusWaitEmptyTimeout);
          break;
        }
        mbar_expect_tx(do_full, kTileBytes);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) tma_load_2d(sDO + c * kChunkBytes, &tmDO, do_full, head * D + c * 64, row);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = mbar_wait(kv_full, 0);
      if (!ok) report_status(p.status, kStatusWaitFullTimeout);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aDO = smem_u32(sDO), aDS = smem_u32(sDS);
      const auto need = [&](uint64_t* bar, uint32_t parity, int code) {
        if (!mbar_wait(bar, parity)) {
          report_status(p.status, code);
          return false;
        }
        tc_fence_after();
        return true;
      };
      const auto score = [&](int it) {  // S^T = K Q^T
        const uint32_t aQ = smem_u32(sQ + (it & 1) * kTileBytes);
        if (!need(&q_full[it & 1], (it >> 1) & 1, kStatusWaitFullTimeout)) return false;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * kChunkBytes + (k % 4) * 32;
          tc_mma_f16(tmem_R1, umma_smem_desc(aK + off, 16, 1024), umma_smem_desc(aQ + off, 16, 1024), kIdescST, k > 0 ? 1u : 0u);
        }
        tc_commit(s_full);
        return true;
      };
      const auto grad_p = [&](int it) {  // dP^T = V dO^T
        if (!need(do_full, it & 1, kStatusWaitFullTimeout)) return false;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * kChunkBytes + (k % 4) * 32;
          tc_mma_f16(tmem_R2, umma_smem_desc(aV + off, 16, 1024), umma_smem_desc(aDO + off, 16, 1024), kIdescST, k > 0 ? 1u : 0u);
        }
        tc_commit(dp_full);
        return true;
      };
      if (ok && n_it > 0) ok = score(0) && grad_p(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t aQ = smem_u32(sQ + (it & 1) * kTileBytes);
        // dV += P^T dO   (A: P^T packed bf16 in R1, B: dO as [N = D, K = queries], MN-major)
        if (!need(p_ready, it & 1, kStatusWaitTmemFullTimeout)) break;
#pragma unroll
        for (int k = 0; k < kT / 16; ++k)
          tc_mma_f16_ts(tmem_dV, tmem_R1 + (k & 3) * 8 + (k >> 2) * 64, umma_smem_desc(aDO + k * 2048, kChunkBytes, 1024), kIdescKV,
                        (it > 0 || k > 0) ? 1u : 0u);
        tc_commit(dv_done);
        if (it + 1 < n_it && !score(it + 1)) break;
        // dQ = dS K      (A: dS^T tile in shared memory read MN-major, B: K as [N = D, K = keys], MN-major)
        if (!need(ds_ready, it & 1, kStatusWaitTmemFullTimeout)) break;
#pragma unroll
        for (int k = 0; k < kT / 16; ++k)
          tc_mma_f16(tmem_R2, umma_smem_desc(aDS + k * 2048, kChunkBytes, 1024),
                     umma_smem_desc(aK + k * 2048, kChunkBytes, 1024), kIdescDQ, k > 0 ? 1u : 0u);
        tc_commit(dq_full);
        // dK += dS^T Q   (the same tile read K-major)
#pragma unroll
        for (int k = 0; k < kT / 16; ++k)
          tc_mma_f16(tmem_dK, umma_smem_desc(aDS + (k >> 2) * kChunkBytes + (k & 3) * 32, 16, 1024),
                     umma_smem_desc(aQ + k * 2048, kChunkBytes, 1024), kIdescKV, (it > 0 || k > 0) ? 1u : 0u);
        tc_commit(&q_empty[it & 1]);
        if (it + 1 < n_it) ok = need(dq_read, it & 1, kStatusWaitTmemEmptyTimeout) && grad_p(it + 1);
      }
      tc_commit(all_done);
    }
  } else {
    // Compute warps: thread = one key row and half of the queries (P^T / dS^T); for the dQ read-out, one query row and half
    // of its columns.
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const int kj = k0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = true;
    // the thread's share of a step's row statistics, requested while the step before is in its products
    const auto row_stat = [&](int it) {
      const int hg = it / n_q, qi = k0 + (it - hg * n_q) * kT + r;
      if (it >= n_it || qi >= seq_len) return part == 0 ? INFINITY : 0.f;
      return (part == 0 ? p.lse : p.delta)[(long long)(head0 + hg) * p.T + seq_start + qi];
    };
    float stat = row_stat(0);
    constexpr int kMine = D / 64;  // 32-column pieces of dQ that this warp takes out
    static_assert(kMine <= 2, "the first piece goes out at once, the second behind the next step's exponentials");
    uint32_t late[32];
    // Piece c of step it's dQ, from registers through 32 rows x 128 bytes of shared memory per warp. Rows past the sequence go out as
    // zeros: the product has 0 there, or NaN where K is not finite, and the next sequence is not to see it. Cleared in shared
    // memory, which costs less than a select on every value.
    const auto send_dq = [&](const uint32_t (&o)[32], int it, int c) {
      const int hg = it / n_q, q0 = k0 + (it - hg * n_q) * kT;
      uint8_t* buf = sOut + (warp - 2) * 4096;
      if (lane == 0) bulk_wait_read<0>();  // the piece before, sent half a step ago
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(buf + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_uint4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
      if (q0 + r >= seq_len) {
#pragma unroll 1
        for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(buf + lane * 128 + u * 16) = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && q0 + quarter * 32 < seq_len) {
        tma_reduce_add_2d(&tmDQ, buf, (head0 + hg) * D + (part * kMine + c) * 32, seq_start + q0 + quarter * 32);
        bulk_commit();
      }
    };
    for (int it = 0; it < n_it; ++it) {
      const int hg = it / n_q, qt = it - hg * n_q;
      const int q0 = k0 + qt * kT;
      const int b = it & 1;
      if (part == 0) sLse[b * kT + r] = -(stat * 1.4426950408889634f);
      else sDelta[b * kT + r] = -stat;
      named_bar_sync(1, 256);
      if (!mbar_wait(s_full, it & 1)) {
        report_status(p.status, kStatusWaitTmemFullTimeout);
        ok = false;
        break;
      }
      tc_fence_after();
      const bool diag = (qt == 0);
      const float2 scale2 = make_float2(p.scale, p.scale), scale_log2 = make_float2(p.scale_log2, p.scale_log2);
      float pr[2][32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = part * 2 + h;
        uint32_t sv[32], pk[16];
        tmem_ld_32x32(tmem_R1 + lane_off + c * 32, sv);
        tc_wait_ld();
#pragma unroll
        for (int i4 = 0; i4 < 32; i4 += 4) {
          const float4 ml = *reinterpret_cast<const float4*>(sLse + b * kT + c * 32 + i4);
#pragma unroll
          for (int i = i4; i < i4 + 4; i += 2) {
            const int qa = c * 32 + i;
            const float2 z = fma2(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), scale_log2,
                                  i == i4 ? make_float2(ml.x, ml.y) : make_float2(ml.z, ml.w));
            float e0 = exp2f(z.x), e1 = exp2f(z.y);
            if (diag) {
              if (kj > q0 + qa) e0 = 0.f;
              if (kj > q0 + qa + 1) e1 = 0.f;
            }
            pr[h][i] = e0;
            pr[h][i + 1] = e1;
            pk[i / 2] = pack_bf16x2(e0, e1);
          }
        }
        tmem_st_32x16(tmem_R1 + lane_off + part * 64 + h * 16, pk);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if constexpr (kMine > 1) {  // the later half of the step before's dQ
        if (it > 0) send_dq(late, it - 1, 1);
      }

      if (!mbar_wait(dp_full, it & 1)) {
        report_status(p.status, kStatusWaitTmemFullTimeout);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = part * 2 + h;
        uint32_t dp[32], dsk[16];
        tmem_ld_32x32(tmem_R2 + lane_off + c * 32, dp);
        tc_wait_ld();
#pragma unroll
        for (int i4 = 0; i4 < 32; i4 += 4) {
          const float4 md = *reinterpret_cast<const float4*>(sDelta + b * kT + c * 32 + i4);
#pragma unroll
          for (int i = i4; i < i4 + 4; i += 2) {
            const float2 e = make_float2(pr[h][i], pr[h][i + 1]);
            float2 d = mul2(mul2(e, add2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])),
                                         i == i4 ? make_float2(md.x, md.y) : make_float2(md.z, md.w))), scale2);
            if (e.x == 0.f) d.x = 0.f;
            if (e.y == 0.f) d.y = 0.f;
            dsk[i / 2] = pack_bf16x2(d.x, d.y);
          }
        }
        // dS^T row r, queries [32c, 32c+32) into the 128-byte-swizzled [keys x queries] tile.
        uint8_t* rowp = sDS + (c >> 1) * kChunkBytes + r * 128;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int unit = ((c & 1) * 4 + u) ^ (r & 7);
          *reinterpret_cast<uint4*>(rowp + unit * 16) = make_uint4(dsk[u * 4], dsk[u * 4 + 1], dsk[u * 4 + 2], dsk[u * 4 + 3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
      stat = row_stat(it + 1);

      if (!mbar_wait(dq_full, it & 1)) {
        report_status(p.status, kStatusWaitTmemFullTimeout);
        ok = false;
        break;
      }
      tc_fence_after();
      {
        uint32_t first[32];
        tmem_ld_32x32(tmem_R2 + lane_off + (part * kMine) * 32, first);
        if constexpr (kMine > 1) tmem_ld_32x32(tmem_R2 + lane_off + (part * kMine + 1) * 32, late);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_read);
        send_dq(first, it, 0);
      }
    }
    if (ok && n_it > 0) {
      if constexpr (kMine > 1) send_dq(late, n_it - 1, 1);
      if (!mbar_wait(all_done, 0)) {
        report_status(p.status, kStatusWaitTmemFullTimeout);
        ok = false;
      }
      tc_fence_after();
    }
    if (lane == 0) bulk_wait_all<0>();
    if (ok && n_it > 0) {
      const bool valid = kj < seq_len;
      const long long t = (long long)seq_start + kj;
      const uint32_t acc = (part == 0 ? tmem_dV : tmem_dK) + lane_off;
      if (p.pieces > 1) {
        float* out = p.dkv + part_offset<D>(piece, gridDim.y, tile_idx, p.Hkv, (part == 0 ? p.Hkv : 0) + kv_head, quarter) + lane * 4;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(acc + c * 32, o);
          tc_wait_ld();
          if (valid) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(out + (c * 8 + i / 4) * 128) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
          }
        }
      } else {
      // the warps of part 0 write dV, those of part 1 dK, whose columns i and D / 2 + i rotate together
      const auto store32 = [](__nv_bfloat16* dst, const float (&v)[32]) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 w;
          w.x = pack_bf16x2(v[i], v[i + 1]);
          w.y = pack_bf16x2(v[i + 2], v[i + 3]);
          w.z = pack_bf16x2(v[i + 4], v[i + 5]);
          w.w = pack_bf16x2(v[i + 6], v[i + 7]);
          *reinterpret_cast<uint4*>(dst + i) = w;
        }
      };
      __nv_bfloat16* out = part == 0 ? p.dv + t * p.ld_dv + p.dv_col0 + (long long)kv_head * D : p.dk + t * p.ld_dk + p.dk_col0 + (long long)kv_head * D;
#pragma unroll 1
      for (int c = 0; c < D / 64; ++c) {
        uint32_t lo[32], hi[32];
        tmem_ld_32x32(acc + c * 32, lo);
        tmem_ld_32x32(acc + D / 2 + c * 32, hi);
        tc_wait_ld();
        if (valid) {
          float x1[32], x2[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            x1[i] = __uint_as_float(lo[i]);
            x2[i] = __uint_as_float(hi[i]);
          }
          if (part == 1 && p.rope.pos != nullptr) {
            const long long row = p.rope.row(t) * (D / 2) + c * 32;
#pragma unroll
            for (int i = 0; i < 32; ++i) rope_rotate(x1[i], x2[i], p.rope.cos_t[row + i], -p.rope.sin_t[row + i]);
          }
          store32(out + c * 32, x1);
          store32(out + D / 2 + c * 32, x2);
        }
      }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; one warp per (t, h).
__global__ void attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                      float* __restrict__ delta, int T, int Hq, int D, long long ldo, long long lddo) {
  pdl_wait();
  pdl_launch();
  const long long w = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)T * Hq) return;
  const int lane = threadIdx.x & 31;
  const int t = (int)(w / Hq), h = (int)(w % Hq);
  const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(o + (long long)t * ldo + (long long)h * D);
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(d_o + (long long)t * lddo + (long long)h * D);
  float acc = 0.f;
  for (int i = lane; i < D / 2; i += 32) {
    const float2 x = __bfloat1622float2(a[i]);
    const float2 y = __bfloat1622float2(b[i]);
    acc += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (lane == 0) delta[(long long)h * T + t] = acc;
}

// out (bf16, pitch ld, `heads` heads) = acc (fp32, pitch lda), rotated back where `rope` says so: a thread converts four columns of
// each half of a head.
__global__ void attn_bwd_finalize_kernel(const float* __restrict__ acc, long long lda, __nv_bfloat16* __restrict__ out, long long ld, long long T,
                                         int heads, int D, const AttnRope rope) {
  pdl_wait();
  pdl_launch();
  const int per_head = D / 8;
  const long long total = T * heads * per_head;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(i % per_head) * 4;
    const long long th = i / per_head;
    const long long t = th / heads;
    const int col = (int)(th % heads) * D + j;
    float4 a = __ldcs(reinterpret_cast<const float4*>(acc + t * lda + col));
    float4 b = __ldcs(reinterpret_cast<const float4*>(acc + t * lda + col + D / 2));
    if (rope.pos != nullptr) {
      const long long row = rope.row(t) * (D / 2) + j;
      const float4 c = *reinterpret_cast<const float4*>(rope.cos_t + row), s = *reinterpret_cast<const float4*>(rope.sin_t + row);
      rope_rotate(a.x, b.x, c.x, -s.x);
      rope_rotate(a.y, b.y, c.y, -s.y);
      rope_rotate(a.z, b.z, c.z, -s.z);
      rope_rotate(a.w, b.w, c.w, -s.w);
    }
    __nv_bfloat16* d = out + t * ld + col;
    *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
    *reinterpret_cast<uint2*>(d + D / 2) = make_uint2(pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
}

// dK and dV (bf16) from the pieces' parts, summed in the order of the pieces, K rotated back where `rope` says so. A block takes one
// part (32 rows of one tile, blockIdx.z: quarter) of one head (blockIdx.y: the heads of K, then those of V); a thread converts 16
// columns of each half of a head, so that a warp reads whole lines and writes whole sectors.
template <int D>
__global__ void __launch_bounds__(D)
attn_bwd_finalize_dkv_kernel(const float* __restrict__ acc, int pieces, const int4* __restrict__ tiles, __nv_bfloat16* __restrict__ dk, long long ld_dk,
                             __nv_bfloat16* __restrict__ dv, long long ld_dv, int Hkv, const AttnRope rope) {
  pdl_wait();
  pdl_launch();
  const int4 tile = tiles[blockIdx.x];
  const int lane = threadIdx.x & 31, j = (threadIdx.x >> 5) * 16, head = blockIdx.y;  // D / 32 warps of 16 columns each
  const int kj = tile.z + blockIdx.z * 32 + lane;
  if (kj >= tile.y) return;
  const bool is_k = head < Hkv;
  const long long t = (long long)tile.x + kj;
  float a[16] = {}, b[16] = {};
#pragma unroll 2
  for (int q = 0; q < pieces; ++q) {
    const float* src = acc + part_offset<D>(q, gridDim.x, blockIdx.x, Hkv, head, blockIdx.z) + lane * 4;
    float4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = __ldcs(reinterpret_cast<const float4*>(src + (j / 4 + i) * 128));
      y[i] = __ldcs(reinterpret_cast<const float4*>(src + ((j + D / 2) / 4 + i) * 128));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[4 * i] += x[i].x; a[4 * i + 1] += x[i].y; a[4 * i + 2] += x[i].z; a[4 * i + 3] += x[i].w;
      b[4 * i] += y[i].x; b[4 * i + 1] += y[i].y; b[4 * i + 2] += y[i].z; b[4 * i + 3] += y[i].w;
    }
  }
  if (is_k && rope.pos != nullptr) {
    const long long row = rope.row(t) * (D / 2) + j;
#pragma unroll
    for (int i = 0; i < 16; ++i) rope_rotate(a[i], b[i], rope.cos_t[row + i], -rope.sin_t[row + i]);
  }
  __nv_bfloat16* d = (is_k ? dk + t * ld_dk + head * D : dv + t * ld_dv + (head - Hkv) * D) + j;
#pragma unroll
  for (int i = 0; i < 16; i += 8) {
    *reinterpret_cast<uint4*>(d + i) = make_uint4(pack_bf16x2(a[i], a[i + 1]), pack_bf16x2(a[i + 2], a[i + 3]), pack_bf16x2(a[i + 4], a[i + 5]), pack_bf16x2(a[i + 6], a[i + 7]));
    *reinterpret_cast<uint4*>(d + D / 2 + i) = make_uint4(pack_bf16x2(b[i], b[i + 1]), pack_bf16x2(b[i + 2], b[i + 3]), pack_bf16x2(b[i + 4], b[i + 5]), pack_bf16x2(b[i + 6], b[i + 7]));
  }
}

void finalize(const float* acc, long long lda, void* out, long long ld, int T, int heads, int D, const AttnRope& rope, cudaStream_t s) {
  const long long blocks = ((long long)T * heads * (D / 8) + 255) / 256;
  launch_kernel(attn_bwd_finalize_kernel, dim3((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0, s, "attn_bwd_finalize", acc, lda,
                (__nv_bfloat16*)out, ld, (long long)T, heads, D, rope);
}

template <int D>
void launch_bwd_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                  const CUtensorMap& tdq, const AttnBwdParams& p, int n_tiles, int Hkv, cudaStream_t s) {
  constexpr int smem = 5 * kT * D * 2 + kT * kT * 2 + 8 * 4096 + 4 * kT * 4 + 128;
  auto kernel = attn_bwd_kernel<D>;
  AGRPO_SET_MAX_DYN_SMEM(kernel, smem, "attn_bwd smem attr");
  dim3 grid(Hkv * p.pieces, n_tiles);
  launch_kernel(kernel, grid, dim3(kBwdThreads), smem, s, "attn_bwd launch", tq, tk, tv, tdo, tdq, p);
}

}  // namespace

// CTAs over which the query heads of a (key tile, kv head) are dealt: enough for about four CTAs per SM, so that the longest of them
// (all query tiles of the longest sequence) is a small part of an SM's share. 12 query and 2 kv heads, us with one piece and with as
// many as this rule says, L2 flushed: one sequence of 759 tokens 130 and 52 (6 pieces), of 2600 404 and 105 (6), of 8000 1187 and 618 (5), 11
// of 250 to 8575 (17341) 841 and 606 (3). Sequences of one length lose: 19 of 330 112 and 122 (6), 40 of 330 169 and 193 (3); 8 of 4096
// 1281 to 1588 and 1316 to 1710 (2), where runs differ more than the choices. The rule goes by the count of tiles alone, which does not
// tell these from the others; the packer knows the lengths, a rule by them is not built. From 592 CTAs on nothing is split.
int attn_bwd_pieces(int n_tiles, int Hq, int Hkv, int num_sms) {
  const long long ctas = (long long)n_tiles * Hkv;
  if (ctas <= 0) return 1;
  const long long want = (4 * num_sms + ctas - 1) / ctas, group = Hq / Hkv;
  return (int)(want < 1 ? 1 : want < group ? want : group);
}

void launch_attn_varlen_bwd(const void* q, long long ldq, int q_cols, const void* k, long long ldk, int k_cols,
                            const void* v, long long ldv, int v_cols, int q_col0, int k_col0, int v_col0, const void* out,
                            long long ldo, const void* dout, long long lddo, const float* lse, float* delta, float* dq_acc,
                            void* dq, long long ld_dq, void* dk, long long ld_dk, int dk_col0, void* dv, long long ld_dv,
                            int dv_col0, const int* tiles, int n_tiles, int T, int Hq, int Hkv, int D, float softmax_scale,
                            int* status, cudaStream_t s, const AttnRope& rope, int pieces, float* dkv_acc) {
  if (n_tiles == 0 || T == 0) return;
  if (D != 64 && D != 128) throw std::runtime_error("attn_varlen_bwd: head_dim must be 64 or 128");
  {
    const long long warps = (long long)T * Hq;
    launch_kernel(attn_bwd_delta_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, s, "attn_bwd_delta", (const __nv_bfloat16*)out,
                  (const __nv_bfloat16*)dout, delta, T, Hq, D, ldo, lddo);
  }
  check_cuda(cudaMemsetAsync(dq_acc, 0, (size_t)T * Hq * D * sizeof(float), s), "attn_bwd dq memset");
  const CUtensorMap tq = make_tmap_2d(q, q_cols, T, ldq, 64, kT);
  const CUtensorMap tk = make_tmap_2d(k, k_cols, T, ldk, 64, kT);
  const CUtensorMap tv = make_tmap_2d(v, v_cols, T, ldv, 64, kT);
  const CUtensorMap tdo = make_tmap_2d(dout, (uint64_t)Hq * D, T, lddo, 64, kT);
  const CUtensorMap tdq = make_tmap_2d(dq_acc, (uint64_t)Hq * D, T, (uint64_t)Hq * D, 32, 32, 4);
  AttnBwdParams p;
  p.tiles = reinterpret_cast<const int4*>(tiles);
  p.lse = lse;
  p.delta = delta;
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.ld_dk = ld_dk;
  p.ld_dv = ld_dv;
  p.dk_col0 = dk_col0;
  p.dv_col0 = dv_col0;
  p.T = T;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.group = Hq / Hkv;
  p.pieces = pieces;
  p.dkv = dkv_acc;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.scale = softmax_scale;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.rope = rope;
  p.status = status;
  if (D == 128) launch_bwd_t<128>(tq, tk, tv, tdo, tdq, p, n_tiles, Hkv, s);
  else          launch_bwd_t<64>(tq, tk, tv, tdo, tdq, p, n_tiles, Hkv, s);
  finalize(dq_acc, (long long)Hq * D, dq, ld_dq, T, Hq, D, rope, s);
  if (pieces > 1)
    launch_kernel(D == 128 ? attn_bwd_finalize_dkv_kernel<128> : attn_bwd_finalize_dkv_kernel<64>, dim3(n_tiles, 2 * Hkv, 4), dim3(D), 0, s,
                  "attn_bwd_finalize_dkv", (const float*)dkv_acc, pieces, p.tiles, p.dk + dk_col0, ld_dk, p.dv + dv_col0, ld_dv, Hkv, rope);
}

}  // namespace agrpo
