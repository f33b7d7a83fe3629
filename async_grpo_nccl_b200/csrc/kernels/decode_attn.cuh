// Paged-KV decode attention (one query token per sequence) as a device function, shared by the stand-alone
// kernel of the rollout engine and by the persistent decode-layers kernel.
#pragma once
#include <cuda_bf16.h>

#include "../common/ptx.cuh"
#include "decode_sync.cuh"

namespace agrpo {

namespace {

// ------------------------------------------------------------------------------------------------
// Paged decode attention (one query token per sequence), D = 128, block_size = 16, G = Hq/Hkv <= 8.
// CTA = (split, kv head, sequence), 4 warps; a warp owns whole 16-token blocks: cp.async double
// buffering into swizzled shared memory, QK^T and PV on mma.sync m16n8k16 with the query heads of the
// group as the (zero-padded) M rows, online softmax in registers. Warps and splits are merged with
// the usual (max, sum, O) rule.
// ------------------------------------------------------------------------------------------------
constexpr int kDecD = 128;
constexpr int kDecBlock = 16;
constexpr int kDecWarps = 4;

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) { cp_async16(smem_u32(smem_dst), gsrc); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem) { ldmatrix_x4(r, smem_u32(smem)); }
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem) { ldmatrix_x4_trans(r, smem_u32(smem)); }
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct DecodeParams {
  const __nv_bfloat16* q;   // [B, row pitch ldq], head h at column q_col0 + h*D
  long long ldq;
  int q_col0;
  const __nv_bfloat16* k_cache;
  const __nv_bfloat16* v_cache;
  const int* block_tables;  // [B, max_blocks]
  const int* seq_lens;      // [B] tokens in the cache including the current one
  int max_blocks;
  int Hq, Hkv, G;
  float scale_log2;
  int splits;
  __nv_bfloat16* out;       // [B, ldo]
  long long ldo;
  float* part_o;            // [B, Hkv, splits, 8, D]
  float* part_ml;           // [B, Hkv, splits, 8, 2]
  int num_cache_blocks;
  int* status;
  int* tickets;             // [B, Hkv] zero-initialised arrival counters, or nullptr: the last split CTA to finish merges
};

// Shared-memory tile of one 16-token block: 16 rows x 256 bytes, 16-byte chunk c of row r stored at c ^ (r & 7). Tiles start on
// 256 bytes, so that chunk c ^ d of a row is at the address of chunk c with d << 4 flipped.
__device__ __forceinline__ uint32_t tile_chunk(uint32_t tile, int row, int chunk) {
  return tile + row * 256 + ((chunk ^ (row & 7)) << 4);
}

// 128 threads (4 warps) work on one (split, kv head, sequence) item; `dsm` is shared memory that they own for the duration of
// the call, `warp` in [0, 4) and `tid` in [0, 128) index the caller's threads. Threads synchronise on named barrier 1 (128
// threads), so the function may be called by a subset of a larger CTA; a caller that loops over items synchronises between them.
__device__ __forceinline__ void dec_bar_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// STAGES = K/V blocks a warp keeps in shared memory (one being consumed, STAGES - 1 in flight): dsm must hold
// 4 * STAGES * 8 KB. A decode item is a chain of block loads, so its time is (blocks per warp) x (load latency) /
// (loads in flight).
// `cache_off`: elements from the caches' start to this layer's. `p` is best a kernel parameter: as a local struct it takes
// 30 registers.
// ready() returns once the query row and the newest token's cache row are visible to the calling warp. The first blocks of older
// tokens are requested before it: they do not depend on this layer.
// emit(g, d, acc, M, L): weighted sum, maximum and denominator of head g at dim d over this split's tokens.
template <int STAGES, class Ready, class Emit>
__device__ __forceinline__ void paged_decode_partial(const DecodeParams& p, long long cache_off, int split, int kvh, int b,
                                                     uint8_t* dsm, int warp, int tid, Ready&& ready, Emit&& emit) {
  const int lane = tid & 31;
  const int seq_len = p.seq_lens[b];
  const int n_blocks = (seq_len + kDecBlock - 1) / kDecBlock;
  const int blk_begin = share(n_blocks, split, p.splits);
  const int blk_end = share(n_blocks, split + 1, p.splits);
  // per-warp staging: STAGES x (K tile 4 KB + V tile 4 KB)
  const uint32_t wbuf = smem_u32(dsm) + warp * (STAGES * 8192);
  const int* table = p.block_tables + (long long)b * p.max_blocks;

  // Tile j of this warp: K (even j) or V (odd j) of its block j / 2, in slot j % (2 STAGES).
  constexpr int kSlots = 2 * STAGES;
  const int my0 = blk_begin + warp;
  const int n_mine = my0 < blk_end ? (blk_end - my0 + kDecWarps - 1) / kDecWarps : 0;
  // Lane k holds the cache block of this warp's block 32 n + k: a load of the table in front of every tile is an L2 round trip
  // in the chain (600 cycles where acquires keep emptying the L1).
  int pages = 0;
  auto load_pages = [&](int first) {
    const int blk = my0 + (first + lane) * kDecWarps;
    pages = blk < blk_end ? table[blk] : 0;
    if (pages < 0 || pages >= p.num_cache_blocks) {
      report_status(p.status, kStatusBadIndex);
      pages = 0;
    }
  };
  load_pages(0);
  // tile j, whose block is one of the 32 that `pages` holds
  auto issue_tile = [&](int j) {
    const int phys = __shfl_sync(0xffffffffu, pages, (j >> 1) & 31);
    const __nv_bfloat16* src = ((j & 1) ? p.v_cache : p.k_cache) + cache_off + ((long long)phys * p.Hkv + kvh) * kDecBlock * kDecD;
    // 256 chunks of 16 bytes per tile: two rows at a time
    const uint32_t dst = tile_chunk(wbuf + (j % kSlots) * 4096, lane >> 4, lane & 15);
    src += lane * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) cp_async16((dst ^ (((2 * i) & 7) << 4)) + i * 512, src + i * 2 * kDecD);
  };

  // One commit group per tile (empty when there is nothing left to load), so that "at most n groups pending" always names the
  // same tile. The first 2 STAGES - 1 tiles now: the scores of block i + 1 are computed before block i's values are added
  // up, so K runs one block ahead of V.
  bool late = false;  // the newest token's block is among the first ones
#pragma unroll 1
  for (int j = 0; j < kSlots - 1; ++j) {
    const int blk = my0 + (j >> 1) * kDecWarps;
    if (blk < blk_end) {
      if (blk == n_blocks - 1) late = true;
      else issue_tile(j);
    }
    cp_async_commit();
  }
  ready();
  if (late) {
    const int j0 = (n_blocks - 1 - my0) / kDecWarps * 2;
    issue_tile(j0);
    if (j0 + 1 < kSlots - 1) issue_tile(j0 + 1);
    cp_async_commit();
    cp_async_wait<0>();
  }

  // Q fragments (A operand, rows = query heads of this kv head, zero above G), pre-scaled later in fp32.
  uint32_t qa[kDecD / 16][2];
  {
    const int g = lane >> 2;
    const __nv_bfloat16* qrow = p.q + (long long)b * p.ldq + p.q_col0 + (long long)(kvh * p.G + g) * kDecD;
#pragma unroll
    for (int kk = 0; kk < kDecD / 16; ++kk) {
      const int c = kk * 16 + (lane & 3) * 2;
      // L2 loads: inside a persistent kernel the query row was written by another SM during this launch, and this SM
      // may still hold the previous layer's row at the same address in its L1
      qa[kk][0] = (g < p.G) ? __ldcg(reinterpret_cast<const uint32_t*>(qrow + c)) : 0u;
      qa[kk][1] = (g < p.G) ? __ldcg(reinterpret_cast<const uint32_t*>(qrow + c + 8)) : 0u;
    }
  }
  float o[kDecD / 8][2];
#pragma unroll
  for (int n = 0; n < kDecD / 8; ++n) o[n][0] = o[n][1] = 0.f;
  float m = -INFINITY, l = 0.f;

  // S = Q K^T of a block's 16 tokens, dims 16 kk .. 16 kk + 15: two n-tiles of 8 tokens.
  auto k_tile = [&](int i) {
    return tile_chunk(wbuf + ((2 * i) % kSlots) * 4096, (lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1);
  };
  auto score_step = [&](uint32_t kt, int kk, float (&a)[4], float (&b)[4]) {
    uint32_t kb[4];
    ldmatrix_x4(kb, kt ^ (kk << 5));
    mma_16816(a, qa[kk][0], 0u, qa[kk][1], 0u, kb[0], kb[1]);
    mma_16816(b, qa[kk][0], 0u, qa[kk][1], 0u, kb[2], kb[3]);
  };
  float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
  if (n_mine > 0) {
    cp_async_wait<kSlots - 2>();  // K of the first block
    __syncwarp();
    const uint32_t kt = k_tile(0);
#pragma unroll
    for (int kk = 0; kk < kDecD / 16; ++kk) score_step(kt, kk, s0, s1);
  }
  // Live at the start of iteration i: V of block i, K of block i + 1; the slot behind them is refilled, then the one of K i.
  for (int i = 0; i < n_mine; ++i) {
    __syncwarp();  // every lane has read K of block i and V of block i - 1
    const int my = my0 + i * kDecWarps;
    {
      const int j = 2 * i + kSlots - 1;  // V of block i + STAGES - 1, K of block i + STAGES
      if (my + (STAGES - 1) * kDecWarps < blk_end) issue_tile(j);
      cp_async_commit();
      if (my + STAGES * kDecWarps < blk_end) {
        if (((i + STAGES) & 31) == 0) load_pages(i + STAGES);
        issue_tile(j + 1);
      }
      cp_async_commit();
    }
    // scores of head lane/4 for tokens {2i, 2i+1, 8+2i, 9+2i}, i = lane%4
    const int tok0 = my * kDecBlock + (lane & 3) * 2;
    float sc[4] = {s0[0] * p.scale_log2, s0[1] * p.scale_log2, s1[0] * p.scale_log2, s1[1] * p.scale_log2};
    if (tok0 >= seq_len) sc[0] = -INFINITY;
    if (tok0 + 1 >= seq_len) sc[1] = -INFINITY;
    if (tok0 + 8 >= seq_len) sc[2] = -INFINITY;
    if (tok0 + 9 >= seq_len) sc[3] = -INFINITY;
    float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m, mx);
    const float alpha = (m == -INFINITY) ? 0.f : exp2f(m - m_new);
    const float base = (m_new == -INFINITY) ? 0.f : m_new;
    float pr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) pr[k] = exp2f(sc[k] - base);
    float ps = pr[0] + pr[1] + pr[2] + pr[3];
    ps += __shfl_xor_sync(0xffffffffu, ps, 1);
    ps += __shfl_xor_sync(0xffffffffu, ps, 2);
    l = l * alpha + ps;
    m = m_new;
    const uint32_t pa0 = pack_bf16x2(pr[0], pr[1]);
    const uint32_t pa2 = pack_bf16x2(pr[2], pr[3]);
    cp_async_wait<kSlots - 2>();  // up to K of block i + 1
    __syncwarp();
    const uint32_t kt = k_tile(i + 1);
    const uint32_t vt = tile_chunk(wbuf + ((2 * i + 1) % kSlots) * 4096, (lane & 7) + (((lane >> 3) & 1) << 3), lane >> 4);
#pragma unroll
    for (int k = 0; k < 4; ++k) s0[k] = s1[k] = 0.f;
    // O += P V of this block (V^T fragments through transposing ldmatrix, two n-tiles of 8 dims per instruction) between the
    // steps of the next block's scores, which are a chain. After the last block those are computed from a stale tile and unused.
#pragma unroll
    for (int n2 = 0; n2 < kDecD / 16; ++n2) {
      uint32_t vb[4];
      ldmatrix_x4_trans(vb, vt ^ (n2 << 5));
      score_step(kt, n2, s0, s1);
      float c0[4] = {o[n2 * 2][0] * alpha, o[n2 * 2][1] * alpha, 0.f, 0.f};
      float c1[4] = {o[n2 * 2 + 1][0] * alpha, o[n2 * 2 + 1][1] * alpha, 0.f, 0.f};
      mma_16816(c0, pa0, 0u, pa2, 0u, vb[0], vb[1]);
      mma_16816(c1, pa0, 0u, pa2, 0u, vb[2], vb[3]);
      o[n2 * 2][0] = c0[0];
      o[n2 * 2][1] = c0[1];
      o[n2 * 2 + 1][0] = c1[0];
      o[n2 * 2 + 1][1] = c1[1];
    }
  }

  // Merge the four warps through shared memory (reusing the staging area after everyone is done).
  dec_bar_sync();
  float* mo = reinterpret_cast<float*>(dsm);           // [warps][8][D]
  float* mml = mo + kDecWarps * 8 * kDecD;             // [warps][8][2]
  float* fin = mml + kDecWarps * 8 * 2;                // [8][8]: weights of the four warps, maximum, denominator
  {
    const int g = lane >> 2;
#pragma unroll
    for (int n = 0; n < kDecD / 8; ++n) {
      const int d = n * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(mo + (warp * 8 + g) * kDecD + d) = make_float2(o[n][0], o[n][1]);
    }
    if ((lane & 3) == 0) {
      mml[(warp * 8 + g) * 2] = m;
      mml[(warp * 8 + g) * 2 + 1] = l;
    }
  }
  dec_bar_sync();
  if (warp == 0) {  // a lane for each of 8 heads x 4 warps
    const int g = lane >> 2;
    float M = -INFINITY, L = 0.f, mine = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, mml[(w * 8 + g) * 2]);
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float mw = mml[(w * 8 + g) * 2];
      const float wgt = (mw == -INFINITY) ? 0.f : exp2f(mw - M);
      L += mml[(w * 8 + g) * 2 + 1] * wgt;
      if (w == (lane & 3)) mine = wgt;
    }
    fin[g * 8 + (lane & 3)] = mine;
    if ((lane & 3) == 0) {
      fin[g * 8 + 4] = M;
      fin[g * 8 + 5] = L;
    }
  }
  dec_bar_sync();
  static_assert(kDecD == kDecWarps * 32, "a thread per output dim");
#pragma unroll 2
  for (int g = 0; g < p.G; ++g) {
    const float4 wgt = *reinterpret_cast<const float4*>(fin + g * 8);
    const float2 ml = *reinterpret_cast<const float2*>(fin + g * 8 + 4);
    float acc = 0.f;
    acc += mo[g * kDecD + tid] * wgt.x;
    acc += mo[(8 + g) * kDecD + tid] * wgt.y;
    acc += mo[(16 + g) * kDecD + tid] * wgt.z;
    acc += mo[(24 + g) * kDecD + tid] * wgt.w;
    emit(g, tid, acc, ml.x, ml.y);
  }
}

// The item as the stand-alone kernel runs it: partial sums to memory, the last split of a (sequence, kv head) merges.
// `s_last` is one shared int.
template <int STAGES, class Ready>
__device__ __forceinline__ void paged_decode_attend(const DecodeParams& p, int split, int kvh, int b, uint8_t* dsm, int warp,
                                                    int tid, int* s_last, Ready&& ready) {
  paged_decode_partial<STAGES>(p, 0, split, kvh, b, dsm, warp, tid, ready, [&](int g, int d, float acc, float M, float L) {
    if (p.splits == 1) {
      p.out[(long long)b * p.ldo + (long long)(kvh * p.G + g) * kDecD + d] = __float2bfloat16(L > 0.f ? acc / L : 0.f);
    } else {
      const long long base = (((long long)b * p.Hkv + kvh) * p.splits + split) * 8 + g;
      p.part_o[base * kDecD + d] = acc;
      if (d == 0) {
        p.part_ml[base * 2] = M;
        p.part_ml[base * 2 + 1] = L;
      }
    }
  });
  // Split-KV merge without a second kernel: every split CTA of a (sequence, kv head) takes a ticket after its
  // partials are visible device-wide; the one that draws the last ticket merges all of them and re-arms the counter.
  if (p.splits > 1 && p.tickets != nullptr) {
    __threadfence();
    dec_bar_sync();
    if (tid == 0) {
      int* t = p.tickets + (long long)b * p.Hkv + kvh;
      const int ticket = atomicAdd(t, 1);
      *s_last = (ticket == p.splits - 1) ? 1 : 0;
      if (*s_last) *t = 0;
    }
    dec_bar_sync();
    if (*s_last) {
      __threadfence();
      // four output dims per thread (16-byte loads of the partial outputs), eight splits at a time with all their loads
      // issued before the first use: they are L2 round trips, and the merging CTA is on the step's critical path
      for (int idx = tid; idx < p.G * (kDecD / 4); idx += kDecWarps * 32) {
        const int g = idx / (kDecD / 4), d = (idx % (kDecD / 4)) * 4;
        const long long base0 = (((long long)b * p.Hkv + kvh) * p.splits) * 8 + g;
        float M = -INFINITY, L = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < p.splits; s0 += 8) {
          float ms[8], ls[8];
          float4 os[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const bool on = s0 + j < p.splits;
            const long long bs = base0 + (long long)(on ? s0 + j : s0) * 8;
            const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + bs * 2));
            ms[j] = on ? ml.x : -INFINITY;
            ls[j] = on ? ml.y : 0.f;
            os[j] = __ldcg(reinterpret_cast<const float4*>(p.part_o + bs * kDecD + d));
          }
          float Mn = M;
#pragma unroll
          for (int j = 0; j < 8; ++j) Mn = fmaxf(Mn, ms[j]);
          const float keep = (M == -INFINITY) ? 0.f : exp2f(M - Mn);
          L *= keep;
          acc.x *= keep; acc.y *= keep; acc.z *= keep; acc.w *= keep;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float w = (ms[j] == -INFINITY) ? 0.f : exp2f(ms[j] - Mn);
            L += ls[j] * w;
            acc.x += os[j].x * w; acc.y += os[j].y * w; acc.z += os[j].z * w; acc.w += os[j].w * w;
          }
          M = Mn;
        }
        uint2 o;  // same expression as the stand-alone combine kernel: both paths give the same bits
        o.x = pack_bf16x2(L > 0.f ? acc.x / L : 0.f, L > 0.f ? acc.y / L : 0.f);
        o.y = pack_bf16x2(L > 0.f ? acc.z / L : 0.f, L > 0.f ? acc.w / L : 0.f);
        *reinterpret_cast<uint2*>(p.out + (long long)b * p.ldo + (long long)(kvh * p.G + g) * kDecD + d) = o;
      }
    }
  }
}

}  // namespace

}  // namespace agrpo
