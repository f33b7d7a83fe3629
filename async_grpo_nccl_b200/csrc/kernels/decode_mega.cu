// All decoder layers of one decode step in ONE persistent launch (one CTA per SM, cooperative launch).
//
// A decode step at small batch is bound by streaming the weights once; as ~140 separate launches each GEMM pays a
// cold start (first TMA round trip, barrier set-up, TMEM allocation) and a tail that are as long as its streaming time.
// Here the weight stream never stops: a dedicated warp issues the TMA loads of every weight tile of every phase of every
// layer in order, limited only by the depth of its shared-memory ring, so the loads of the next phase are in flight
// while the current phase's results are still being reduced. Only the (small) activation loads wait for the phase before.
//
// The GEMMs run "swapped": the weight tile supplies the 128 MMA rows (output features), the batch rows are the MMA N
// dimension (BT = 32 .. 256), so a small batch costs a small MMA and no padding traffic.
//
//   per layer:  qkv = rs(x) * (x . Wqkv'^T) + b, RoPE, KV-cache write      (phase 0, split K)
//               attention over the paged cache, split-KV                     (compute warps)
//               x1  = x + attn . Wo^T, row sums of squares                    (phase 1, split K)
//               act = silu(rs * x1 . Wg'^T) * (rs * x1 . Wu'^T)               (phase 2)
//               x   = x1 + act . Wd^T, row sums of squares                    (phase 3, split K)
//   (W' = weight with the RMSNorm weight folded into its columns, rs = 1 / rms of the row.)
//
// Work item of a GEMM phase = (128-feature tile, K split). Every item writes its fp32 partial tile to a scratch slot
// (L2-resident) and reduces ITS share of the batch rows over the S partials in a fixed order, then applies the epilogue: the
// reduction is spread over all CTAs and its result does not depend on arrival order. Partials are handed over without a flag
// (kNotYet in decode_sync.cuh): fence, arrival counter and load cost three L2 round trips where polling the data costs
// one. A gate / up tile that is not split along K goes from the accumulator to the activation without leaving the CTA. The
// splits of an attention item are merged the same way, heads dealt to the splits. A global counter `done` counts finished
// shares; the activation producer and the compute warps wait for the count that says that the phase before is complete, the
// latter so that row statistics and residuals are in registers when the accumulator is. Attention has warps of its own: in one
// loop with the epilogues its registers spill, and local memory is slow here, since every acquire empties the L1.
//
// The code has to stay small: every role's instructions are needed once a phase, and at 161 KB of them each phase waited for the
// instruction cache (an epilogue of 1.5 us took 5). So loops that run once a layer are not unrolled, and waits poll in one place.
//
// Bound by the chain of hand-offs, not by bytes. 28 layers of 1536 / 8960, a step: 16 rows x 2048 tokens 1.66 ms with arrival
// counters and attention in the compute warps, 1.45 ms so; 32 rows x 1024 tokens 1.65 and 1.42 (weights alone: 0.48). Handing the
// activations over by value as well (polled by the attention warps) gave 1.44 and 1.43: what it saved in fences it lost to the
// polls' traffic.
//
// Every wait is bounded; a wait that runs out records a status code, makes the CTA leave through its normal exit (TMEM
// freed) and the other CTAs follow as soon as they see the status word.
#include <cuda_bf16.h>

#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "../launchers.h"
#include "decode_attn.cuh"
#include "decode_sync.cuh"

namespace agrpo {

namespace {

constexpr int kMegaThreads = 384;  // weights, activations, products, watcher; four compute warps; four attention warps
constexpr int kFT = 128;                    // features per item (MMA M)
constexpr int kMBK = 64;                    // K per stage
constexpr int kWStage = kFT * kMBK * 2;     // 16 KB
constexpr int kCounterWords = 4;

struct MegaPhase {
  int n_groups;  // feature tiles
  int S;         // K splits per tile
  int num_kb;    // K / 64
};

struct MegaParams {
  int L, B, H, Q, QD, F, Hq, Hkv, grid;
  MegaPhase ph[4];
  int att_items, splits;  // att_items: rows x kv heads x splits
  unsigned int per_layer;  // `done` increments per layer
  __nv_bfloat16 *x, *x1, *qkv, *attn, *act;
  const __nv_bfloat16* bqkv;
  long long bqkv_stride;
  sumsq_t* ss;
  int ss_stride;
  float eps, inv_h;
  const float *cos_t, *sin_t;
  int max_pos;
  const int* block_tables;
  int max_blocks;
  const int* seq_lens;
  __nv_bfloat16* cache;
  long long cache_layer_stride, cache_v_off;
  int num_cache_blocks;
  DecodeParams att;
  float* partials;
  unsigned int* done;
  int* status;
  long long* trace;  // optional: clock64 stamps of CTA 0 in layer trace_layer (32 slots), nullptr = off
  int trace_layer;
  int trace_all;     // also record 4 global-timer stamps per CTA (trace must hold 32 + 4 * grid words)
};

__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// per-CTA stamps (global nanosecond timer) behind the 32 slots of CTA 0: trace[32 + 4 * cta + k]
#define MEGA_STAMP_ALL(k)                                                                       \
  do {                                                                                          \
    if (p.trace != nullptr && p.trace_all && l == p.trace_layer) p.trace[32 + 4 * cta + (k)] = global_ns(); \
  } while (0)

#define MEGA_STAMP(slot)                                                                        \
  do {                                                                                          \
    if (p.trace != nullptr && cta == 0 && l == p.trace_layer) p.trace[slot] = clock64();        \
  } while (0)

__device__ __forceinline__ float4 shfl_xor4(float4 v, int m) {
  return make_float4(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m),
                     __shfl_xor_sync(0xffffffffu, v.z, m), __shfl_xor_sync(0xffffffffu, v.w, m));
}
template <int BT>
struct MegaCfg {
  static constexpr int kXStage = BT * kMBK * 2;
  static constexpr int kNSW = 7;
  static constexpr int kXA = 98304;  // activation ring; the attention phase stages K/V tiles here (3 blocks per warp)
  static constexpr int kNSX = (kXA / kXStage) > 8 ? 8 : (kXA / kXStage);
  static constexpr int kAcc = 2;
  static constexpr uint32_t kTmemCols = (kAcc * BT) < 32 ? 32 : (kAcc * BT);
  static constexpr int kEx = 32 * kFT * 4;  // gate / up exchange: 32 rows
  static constexpr int kSmem = kNSW * kWStage + kXA + kEx + 1024 /* barriers */ + 1024 /* alignment */;
  // rows of a share that a warp reduces at a time, and partials of a row requested at a time
  static constexpr int kRU = BT <= 32 ? 1 : 2;
  static constexpr int kNS = BT <= 32 ? 12 : 4;
};

// What the roles of one CTA share.
struct MegaShared {
  uint64_t full_w[8], empty_w[8], full_x[8], empty_x[8], tmem_full[2], tmem_empty[2], xa_bar;
  uint32_t tmem_slot;
  unsigned int seen;     // the value of `done` that this CTA has observed
  unsigned int xa_free;  // layers whose qkv products have read all that they need from the activation ring
};

constexpr int kAttStages = 3;

// Polls until every value of `t` that is wanted has arrived; load(k) and wanted(k) of value k, arrived(value). False when the
// wait ran out.
template <class T, int N, class Load, class Wanted, class Arrived>
__device__ __forceinline__ bool gather_handoff(T (&t)[N], const int* status, Load&& load, Wanted&& wanted, Arrived&& arrived) {
  uint32_t missing = 0;
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (wanted(k)) missing |= 1u << k;
  bool ok = true;
  const long long t0 = clock64();
  int it = 0;
#pragma unroll 1
  while (missing != 0) {  // one copy of the loads
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (missing >> k & 1) t[k] = load(k);
#pragma unroll
    for (int k = 0; k < N; ++k)
      if ((missing >> k & 1) && arrived(t[k])) missing &= ~(1u << k);
    if ((++it & 31) == 0 && (status_set(status) || clock64() - t0 > kWaitBudgetTicks)) {
      report_status(const_cast<int*>(status), kStatusBarrierTimeout);
      ok = false;
      break;
    }
  }
  __syncwarp();
  return ok;
}

// One attention item: this split's share of the tokens of (sequence b, kv head kvh), then, with several splits, heads split,
// split + splits, ... merged over all of them, one warp a head, four dims a lane. False in the lanes whose wait ran out.
__device__ __forceinline__ bool mega_attention_item(const DecodeParams& dp, long long cache_off, int split, int kvh, int b, uint8_t* xa,
                                                    int cw, int tid, const unsigned int* seen, unsigned int qkv_done, long long* trace) {
  const int lane = tid & 31;
  const int splits = dp.splits;
  const long long slot0 = ((long long)b * dp.Hkv + kvh) * splits * 8;
  bool ok = true;
  paged_decode_partial<kAttStages>(
      dp, cache_off, split, kvh, b, xa, cw, tid,
      [&] {
        if (!wait_seen(seen, qkv_done, dp.status)) {
          report_status(dp.status, kStatusPeerFlagTimeout);
          ok = false;
        }
        __syncwarp();
        if (trace != nullptr && tid == 0) trace[24] = clock64();
      },
      [&](int g, int d, float a, float M, float L) {
        if (splits == 1) {
          dp.out[(long long)b * dp.ldo + (long long)(kvh * dp.G + g) * kDecD + d] = __float2bfloat16(L > 0.f ? a / L : 0.f);
        } else {
          const long long s = slot0 + split * 8 + g;
          st_handoff(dp.part_o + s * kDecD + d, a);
          if (d == 0) {
            st_handoff(dp.part_ml + s * 2, M);
            st_handoff(dp.part_ml + s * 2 + 1, L);
          }
        }
      });
  if (trace != nullptr && tid == 0) trace[27] = clock64();
  if (splits == 1) return ok;
  for (int g = split + splits * cw; g < dp.G; g += splits * 4) {
    float M = -INFINITY, L = 0.f;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < splits; s0 += 8) {
      struct Part {
        float4 o;
        float2 ml;
      } v[8];
      auto po = [&](int k) { return reinterpret_cast<float4*>(dp.part_o + (slot0 + (s0 + k) * 8 + g) * kDecD) + lane; };
      auto pm = [&](int k) { return reinterpret_cast<float2*>(dp.part_ml + (slot0 + (s0 + k) * 8 + g) * 2); };
      ok = gather_handoff(v, dp.status, [&](int k) { return Part{ld_handoff4(po(k)), ld_handoff2(pm(k))}; },
                          [&](int k) { return s0 + k < splits; },
                          [](const Part& t) { return has_arrived(t.o) && has_arrived(t.ml.x) && has_arrived(t.ml.y); }) && ok;
      float Mn = M;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (s0 + j < splits) {
          clear_handoff4(po(j));
          if (lane == 0) clear_handoff2(pm(j));
          Mn = fmaxf(Mn, v[j].ml.x);
        }
      const float keep = (M == -INFINITY) ? 0.f : exp2f(M - Mn);
      L *= keep;
      a.x *= keep; a.y *= keep; a.z *= keep; a.w *= keep;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (s0 + j >= splits) continue;
        const float w = (v[j].ml.x == -INFINITY) ? 0.f : exp2f(v[j].ml.x - Mn);
        L += v[j].ml.y * w;
        a.x += v[j].o.x * w; a.y += v[j].o.y * w; a.z += v[j].o.z * w; a.w += v[j].o.w * w;
      }
      M = Mn;
    }
    uint2 o;  // the expression of the stand-alone kernel: both paths give the same bits
    o.x = pack_bf16x2(L > 0.f ? a.x / L : 0.f, L > 0.f ? a.y / L : 0.f);
    o.y = pack_bf16x2(L > 0.f ? a.z / L : 0.f, L > 0.f ? a.w / L : 0.f);
    *reinterpret_cast<uint2*>(dp.out + (long long)b * dp.ldo + (long long)(kvh * dp.G + g) * kDecD + 4 * lane) = o;
  }
  return ok;
}

template <int BT>
__global__ void __launch_bounds__(kMegaThreads, 1)
decode_layers_kernel(const __grid_constant__ CUtensorMap tmWqkv, const __grid_constant__ CUtensorMap tmWo,
                     const __grid_constant__ CUtensorMap tmWgu, const __grid_constant__ CUtensorMap tmWd,
                     const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmAttn,
                     const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmAct, const MegaParams p) {
  using Cfg = MegaCfg<BT>;
  constexpr int NSW = Cfg::kNSW, NSX = Cfg::kNSX;
  constexpr uint32_t kIdesc = umma_idesc_bf16(kFT, BT, 0, 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_ring = smem;
  uint8_t* xa = smem + NSW * kWStage;
  float* ex = reinterpret_cast<float*>(xa + Cfg::kXA);
  MegaShared* sh = reinterpret_cast<MegaShared*>(xa + Cfg::kXA + Cfg::kEx);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = blockIdx.x, G = p.grid;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 8; ++s) {
      mbar_init(&sh->full_w[s], 1);
      mbar_init(&sh->empty_w[s], 1);
      mbar_init(&sh->full_x[s], 1);
      mbar_init(&sh->empty_x[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sh->tmem_full[a], 1);
      mbar_init(&sh->tmem_empty[a], 4);  // the compute warps
    }
    mbar_init(&sh->xa_bar, 128);
    sh->seen = 0;
    sh->xa_free = 0;
    fence_mbar_init();
  }
  if (warp == 3) {
    tmem_alloc(&sh->tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_slot;
  // done-counter value at which the inputs of GEMM phase ph of layer l are complete
  auto target = [&](int l, int ph) -> unsigned int {
    unsigned int t = (unsigned int)l * p.per_layer;
    if (ph >= 1) t += (unsigned int)(p.ph[0].n_groups * p.ph[0].S) + (unsigned int)p.att_items;
    if (ph >= 2) t += (unsigned int)(p.ph[1].n_groups * p.ph[1].S);
    if (ph >= 3) t += (unsigned int)(p.ph[2].n_groups * p.ph[2].S);
    return t;
  };

  // Registers at launch: 384 x 168. What the four single-thread roles do not need goes to the attention warps, whose loop
  // spills at 168 (96 + 168 + 240 = 3 x 168).
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    if (warp == 0) {
      // ================= weight producer: never waits for another CTA =================
      // Tiles in the order in which the products use them (layer, phase, item, K block), limited only by the depth of the ring. (Asking
      // for tiles further on to be brought into L2 costs more than it gives: 8 tiles ahead 1.47 ms a step of 16 rows, none 1.44.)
      if (elect_one()) {
        int st = 0;
        uint32_t par = 0;
        bool ok = true;
#pragma unroll 1
        for (int l = 0; l < p.L && ok; ++l) {
#pragma unroll 1
          for (int ph = 0; ph < 4 && ok; ++ph) {
            const CUtensorMap* map = ph == 0 ? &tmWqkv : ph == 1 ? &tmWo : ph == 2 ? &tmWgu : &tmWd;
            const int S = p.ph[ph].S, nkb = p.ph[ph].num_kb, n_items = p.ph[ph].n_groups * S;
#pragma unroll 1
            for (int item = cta; item < n_items && ok; item += G) {
              const int ft = item / S, ks = item - ft * S;
              const int row = ft * (ph == 2 ? 64 : kFT);
              const int kb1 = share(nkb, ks + 1, S);
#pragma unroll 1
              for (int kb = share(nkb, ks, S); kb < kb1; ++kb) {
                if (!mbar_wait_s(&sh->empty_w[st], par ^ 1, p.status)) {
                  report_status(p.status, kStatusWaitEmptyTimeout);
                  ok = false;
                  break;
                }
                uint8_t* dst = w_ring + st * kWStage;
                mbar_expect_tx(&sh->full_w[st], kWStage);
                // gate / up: 64 gate features on MMA rows 0..63 (the map's box), the matching 64 up features on rows 64..127
                tma_load_3d(dst, map, &sh->full_w[st], kb * kMBK, row, l);
                if (ph == 2) tma_load_3d(dst + 64 * kMBK * 2, map, &sh->full_w[st], kb * kMBK, p.F + row, l);
                if (++st == NSW) {
                  st = 0;
                  par ^= 1;
                }
              }
            }
          }
        }
      }
    } else if (warp == 1) {
      // ================= activation producer: waits for the phase that writes its operand =================
      if (elect_one()) {
        int st = 0;
        uint32_t par = 0;
        bool ok = true;
        // Layer whose attention phase lies between this CTA's last load and the next, -1 if none. A CTA without work items never
        // waits for xa_bar: its compute warps may be several phases of that barrier ahead.
        int staged = -1;
        for (int l = 0; l < p.L && ok; ++l) {
          for (int ph = 0; ph < 4 && ok; ++ph) {
            const CUtensorMap* tm = ph == 0 ? &tmX : ph == 1 ? &tmAttn : ph == 2 ? &tmX1 : &tmAct;
            const int S = p.ph[ph].S, nkb = p.ph[ph].num_kb, n_items = p.ph[ph].n_groups * S;
            if (ph == 1) staged = l;
            bool waited = (l == 0 && ph == 0);
            for (int item = cta; item < n_items && ok; item += G) {
              if (!waited) {
                if (!wait_seen(&sh->seen, target(l, ph), p.status)) {
                  report_status(p.status, kStatusPeerFlagTimeout);
                  ok = false;
                  break;
                }
                fence_proxy_async_all();  // other SMs wrote the operand with ordinary stores; TMA reads it
                waited = true;
              }
              if (staged >= 0) {
                // the attention phase used this ring's memory through the generic proxy: its threads fenced and arrived
                if (!mbar_wait_s(&sh->xa_bar, (uint32_t)(staged & 1), p.status)) {
                  report_status(p.status, kStatusBarrierTimeout);
                  ok = false;
                  break;
                }
                staged = -1;
              }
              const int ft = item / S, ks = item - ft * S;
              const int kb0 = share(nkb, ks, S), kb1 = share(nkb, ks + 1, S);
              for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait_s(&sh->empty_x[st], par ^ 1, p.status)) {
                  report_status(p.status, kStatusWaitEmptyTimeout);
                  ok = false;
                  break;
                }
                mbar_expect_tx(&sh->full_x[st], Cfg::kXStage);
                tma_load_2d(xa + st * Cfg::kXStage, tm, &sh->full_x[st], kb * kMBK, 0);
                if (++st == NSX) {
                  st = 0;
                  par ^= 1;
                }
              }
            }
          }
        }
      }
    } else if (warp == 2) {
      // ================= MMA issuer =================
      if (elect_one()) {
        int sw = 0, sx = 0, acc = 0;
        uint32_t pw = 0, px = 0, pa = 0;
        bool ok = true;
        for (int l = 0; l < p.L && ok; ++l) {
          for (int ph = 0; ph < 4 && ok; ++ph) {
            const int S = p.ph[ph].S, nkb = p.ph[ph].num_kb, n_items = p.ph[ph].n_groups * S;
            for (int item = cta; item < n_items && ok; item += G) {
              const int ft = item / S, ks = item - ft * S;
              const int kb0 = share(nkb, ks, S), kb1 = share(nkb, ks + 1, S);
              if (!mbar_wait_s(&sh->tmem_empty[acc], pa ^ 1, p.status)) {
                report_status(p.status, kStatusWaitTmemEmptyTimeout);
                ok = false;
                break;
              }
              tc_fence_after();
              const uint32_t d_addr = tmem_base + (uint32_t)(acc * BT);
              for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait_s(&sh->full_w[sw], pw, p.status) || !mbar_wait_s(&sh->full_x[sx], px, p.status)) {
                  report_status(p.status, kStatusWaitFullTimeout);
                  ok = false;
                  break;
                }
                tc_fence_after();
                if (kb == kb0) MEGA_STAMP(ph * 6 + 0);
                if (kb == kb0 && ph == 1) MEGA_STAMP_ALL(2);
                if (kb == kb0 && ph == 0) MEGA_STAMP_ALL(3);
                const uint32_t sa = smem_u32(w_ring + sw * kWStage);
                const uint32_t sb = smem_u32(xa + sx * Cfg::kXStage);
#pragma unroll
                for (int k = 0; k < kMBK / 16; ++k)
                  tc_mma_f16(d_addr, umma_smem_desc(sa + k * 32, 16, 1024), umma_smem_desc(sb + k * 32, 16, 1024), kIdesc,
                             (kb > kb0 || k > 0) ? 1u : 0u);
                tc_commit(&sh->empty_w[sw]);
                tc_commit(&sh->empty_x[sx]);
                if (++sw == NSW) {
                  sw = 0;
                  pw ^= 1;
                }
                if (++sx == NSX) {
                  sx = 0;
                  px ^= 1;
                }
              }
              if (!ok) break;
              tc_commit(&sh->tmem_full[acc]);
              MEGA_STAMP(ph * 6 + 1);
              if (++acc == Cfg::kAcc) {
                acc = 0;
                pa ^= 1;
              }
            }
          }
        }
      }
    } else if (warp == 3) {
      // ================= watcher: the only thread of the CTA that polls the global counter =================
      if (elect_one()) {
        bool ok = true;
        for (int l = 0; l < p.L && ok; ++l) {
          for (int step = 0; step < 5 && ok; ++step) {  // inputs of qkv, attention, o, gate / up, down
            const unsigned int want = step == 1 ? (unsigned int)l * p.per_layer + (unsigned int)(p.ph[0].n_groups * p.ph[0].S)
                                                : target(l, step == 0 ? 0 : step - 1);
            if (!wait_counter(p.done, want, p.status)) {
              report_status(p.status, kStatusPeerFlagTimeout);
              ok = false;
            } else {
              st_release_cta(&sh->seen, want);
            }
          }
        }
      }
    }
  } else if (warp < 8) {
    // ================= compute warps: GEMM reductions + epilogues =================
    const int cw = warp - 4;             // TMEM lane quarter (warp % 4)
    const int tid = threadIdx.x - 128;   // 0..127
    const uint32_t lane_off = static_cast<uint32_t>(cw * 32) << 16;
    int acc = 0;
    uint32_t pa = 0;
    bool fail = false;  // this warp's; all compute warps leave together at the next group_bar_or
    bool ok = true;
    const int B = p.B;
    auto wait_done = [&](unsigned int want) {
      if (!wait_seen(&sh->seen, want, p.status)) {
        report_status(p.status, kStatusPeerFlagTimeout);
        fail = true;
      }
      __syncwarp();
    };

    for (int l = 0; l < p.L && ok; ++l) {
      __nv_bfloat16* k_cache = p.cache + (long long)l * p.cache_layer_stride;
      __nv_bfloat16* v_cache = k_cache + p.cache_v_off;
      if (tid == 0) MEGA_STAMP(26);
      for (int ph = 0; ph < 4 && ok; ++ph) {
        // ---------------- GEMM items of this phase ----------------
        const int S = p.ph[ph].S, n_items = p.ph[ph].n_groups * S;
        bool waited = l == 0 && ph == 0;
        for (int item = cta; item < n_items && ok; item += G) {
          const int grp = item / S, ks = item - grp * S;
          if (!waited) wait_done(target(l, ph));
          waited = true;
          const int r0 = share(B, ks, S), r1 = share(B, ks + 1, S);
          constexpr int RU = Cfg::kRU, NS = Cfg::kNS;
          const int b_first = r0 + cw * RU;
          // Row statistics, lengths and the residual of this warp's first rows: requested while the product still runs.
          sumsq_t m_ss[RU];
          int m_len[RU];
          float4 m_rr[RU], m_cs[RU], m_sn[RU];
          int m_blk[RU];
          auto load_meta = [&](int b0) {
#pragma unroll
            for (int j = 0; j < RU; ++j) {
              const int b = (b0 + j < r1) ? b0 + j : r0;
              m_ss[j] = 0;
              m_len[j] = 0;
              m_rr[j] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (b0 < r1) {
                if (ph == 0) {
                  m_ss[j] = ld_sumsq_l2(p.ss + (size_t)(2 * l) * p.ss_stride + b);
                  m_len[j] = p.seq_lens[b];
                } else if (ph == 2) {
                  m_ss[j] = ld_sumsq_l2(p.ss + (size_t)(2 * l + 1) * p.ss_stride + b);
                } else {
                  m_rr[j] = ld_bf16x4((ph == 1 ? p.x : p.x1) + (size_t)b * p.H + grp * kFT + 4 * lane);
                }
              }
            }
            if (ph == 0 && b0 < r1) {  // rotary table entries and the cache block of each row's position
              const bool not_q = grp >= p.Hq;
              const int jr = (4 * lane) & 63;
#pragma unroll
              for (int j = 0; j < RU; ++j) {
                const int b = (b0 + j < r1) ? b0 + j : r0;
                const int pos = m_len[j] > 0 ? m_len[j] - 1 : 0;
                const int pp = pos >= p.max_pos ? p.max_pos - 1 : pos;
                m_cs[j] = *reinterpret_cast<const float4*>(p.cos_t + (size_t)pp * 64 + jr);
                m_sn[j] = *reinterpret_cast<const float4*>(p.sin_t + (size_t)pp * 64 + jr);
                m_blk[j] = (not_q && m_len[j] > 0) ? p.block_tables[(long long)b * p.max_blocks + pos / kDecBlock] : 0;
              }
            }
          };
          const bool direct = ph == 2 && S == 1;
          // direct: statistics of rows 32 c + lane
          auto row_scale = [&](int c) {
            const int b = c * 32 + lane;
            return b < B ? rsqrtf(sumsq_from_fixed(ld_sumsq_l2(p.ss + (size_t)(2 * l + 1) * p.ss_stride + b)) * p.inv_h + p.eps) : 0.f;
          };
          float rs_next = 0.f;
          if (direct) rs_next = row_scale(0);
          float* gbase = p.partials + (size_t)(grp * S) * (BT * kFT);
          // The first pass begins before the product is complete (at least one, also for a warp without rows); one copy of the code.
#pragma unroll 1
          for (int b0 = b_first; b0 == b_first || b0 < r1; b0 += 4 * RU) {
            if (!direct) load_meta(b0);
            if (b0 == b_first) {
              if (!mbar_wait_s(&sh->tmem_full[acc], pa, p.status)) {
                report_status(p.status, kStatusWaitTmemFullTimeout);
                fail = true;
              }
              tc_fence_after();
              if (tid == 0) MEGA_STAMP(ph * 6 + 2);
              float* slot = p.partials + (size_t)item * (BT * kFT);
#pragma unroll 1
              for (int c = 0; c < BT / 32; ++c) {
                if (c * 32 >= B) break;  // padding rows
                uint32_t r[32];
                tmem_ld_32x32(tmem_base + lane_off + (uint32_t)(acc * BT + c * 32), r);
                tc_wait_ld();
                if (!direct) {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    if (c * 32 + i < B) st_handoff(slot + (size_t)(c * 32 + i) * kFT + cw * 32 + lane, __uint_as_float(r[i]));
                  continue;
                }
                // Warps 0 and 1 hold the gate features, 2 and 3 the up features: through shared memory, then a warp takes every fourth
                // row, a lane two features.
                const float rs_mine = rs_next;
                if (c + 1 < BT / 32 && (c + 1) * 32 < B) rs_next = row_scale(c + 1);
                if (c > 0) asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 32; ++i) ex[i * kFT + cw * 32 + lane] = __uint_as_float(r[i]);
                asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll 2
                for (int i = cw; i < 32; i += 4) {
                  const int row = c * 32 + i;
                  if (row >= B) break;
                  const float rs = __shfl_sync(0xffffffffu, rs_mine, i);
                  const float2 gv = *reinterpret_cast<const float2*>(ex + i * kFT + 2 * lane);
                  const float2 uv = *reinterpret_cast<const float2*>(ex + i * kFT + 64 + 2 * lane);
                  const float g0 = gv.x * rs, g1 = gv.y * rs;
                  *reinterpret_cast<uint32_t*>(p.act + (size_t)row * p.F + grp * 64 + 2 * lane) =
                      pack_bf16x2(g0 / (1.f + __expf(-g0)) * (uv.x * rs), g1 / (1.f + __expf(-g1)) * (uv.y * rs));
                }
              }
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&sh->tmem_empty[acc]);
              if (tid == 0) MEGA_STAMP(ph * 6 + 3);
              if (++acc == Cfg::kAcc) {
                acc = 0;
                pa ^= 1;
              }
            }
            if (direct || b0 >= r1) break;
            // ---- my share of the rows: reduce over the S partials, epilogue ----
            float4 v[RU];
            bool on[RU];
#pragma unroll
            for (int j = 0; j < RU; ++j) {
              on[j] = b0 + j < r1;
              v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            for (int s0 = 0; s0 < S; s0 += NS) {
              float4 t[NS * RU];  // split s0 + k / RU of row b0 + k % RU
              auto src = [&](int k) { return reinterpret_cast<float4*>(gbase + ((size_t)(s0 + k / RU) * BT + b0 + k % RU) * kFT) + lane; };
              auto wanted = [&](int k) { return s0 + k / RU < S && b0 + k % RU < r1; };
              if (!gather_handoff(t, p.status, [&](int k) { return ld_handoff4(src(k)); }, wanted, [](const float4& w) { return has_arrived(w); }))
                fail = true;
              if (tid == 0) MEGA_STAMP(ph * 6 + 4);
#pragma unroll
              for (int k = 0; k < NS * RU; ++k)
                if (wanted(k)) {  // fixed order over the splits
                  clear_handoff4(src(k));
                  float4& w = v[k % RU];
                  w.x += t[k].x; w.y += t[k].y; w.z += t[k].z; w.w += t[k].w;
                }
            }
            if (ph == 0) {
              const bool is_q = grp < p.Hq, is_k = !is_q && grp < p.Hq + p.Hkv;
              float4 bb = make_float4(0.f, 0.f, 0.f, 0.f);
              if (p.bqkv != nullptr) bb = ld_bf16x4(p.bqkv + (long long)l * p.bqkv_stride + grp * kFT + 4 * lane);
              const int* len = m_len;
              const int* blk = m_blk;
              const float4* cs = m_cs;
              const float4* sn = m_sn;
#pragma unroll
              for (int j = 0; j < RU; ++j) {
                if (!on[j]) continue;  // warp-uniform
                const int b = b0 + j;
                const float rs = rsqrtf(sumsq_from_fixed(m_ss[j]) * p.inv_h + p.eps);
                float4 w = make_float4(v[j].x * rs + bb.x, v[j].y * rs + bb.y, v[j].z * rs + bb.z, v[j].w * rs + bb.w);
                if (is_q || is_k) {
                  const float4 o = shfl_xor4(w, 16);
                  const float sg = lane < 16 ? -1.f : 1.f;  // lanes < 16 hold x1 (x1 c - x2 s), the others x2 (x2 c + x1 s)
                  w = make_float4(w.x * cs[j].x + sg * o.x * sn[j].x, w.y * cs[j].y + sg * o.y * sn[j].y,
                                  w.z * cs[j].z + sg * o.z * sn[j].z, w.w * cs[j].w + sg * o.w * sn[j].w);
                }
                st_bf16x4(p.qkv + (size_t)b * p.Q + grp * kFT + 4 * lane, w);
                if (!is_q && len[j] > 0) {
                  if (blk[j] < 0 || blk[j] >= p.num_cache_blocks) {
                    report_status(p.status, kStatusBadIndex);
                  } else {
                    const int pos = len[j] - 1;
                    const int h = grp - p.Hq - (is_k ? 0 : p.Hkv);
                    __nv_bfloat16* row = (is_k ? k_cache : v_cache) +
                                         (((long long)blk[j] * p.Hkv + h) * kDecBlock + pos % kDecBlock) * kDecD;
                    st_bf16x4(row + 4 * lane, w);
                  }
                }
              }
            } else if (ph == 2) {
#pragma unroll
              for (int j = 0; j < RU; ++j) {
                if (!on[j]) continue;
                const float rs = rsqrtf(sumsq_from_fixed(m_ss[j]) * p.inv_h + p.eps);
                const float4 u = shfl_xor4(v[j], 16);  // lanes < 16 hold gate features, lanes >= 16 the matching up features
                if (lane < 16) {
                  float4 o;
                  const float g0 = v[j].x * rs, g1 = v[j].y * rs, g2 = v[j].z * rs, g3 = v[j].w * rs;
                  o.x = g0 / (1.f + __expf(-g0)) * (u.x * rs);
                  o.y = g1 / (1.f + __expf(-g1)) * (u.y * rs);
                  o.z = g2 / (1.f + __expf(-g2)) * (u.z * rs);
                  o.w = g3 / (1.f + __expf(-g3)) * (u.w * rs);
                  st_bf16x4(p.act + (size_t)(b0 + j) * p.F + grp * 64 + 4 * lane, o);
                }
              }
            } else {
              __nv_bfloat16* obase = ph == 1 ? p.x1 : p.x;
#pragma unroll
              for (int j = 0; j < RU; ++j) {
                if (!on[j]) continue;
                const float4 w = make_float4(v[j].x + m_rr[j].x, v[j].y + m_rr[j].y, v[j].z + m_rr[j].z, v[j].w + m_rr[j].w);
                st_bf16x4(obase + (size_t)(b0 + j) * p.H + grp * kFT + 4 * lane, w);
                float sq = __fmaf_rn(w.w, w.w, __fmaf_rn(w.z, w.z, __fmaf_rn(w.x, w.x, __fmul_rn(w.y, w.y))));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
                if (lane == 0) sumsq_atomic_add(p.ss + (size_t)(2 * l + (ph == 1 ? 1 : 2)) * p.ss_stride + b0 + j, sq);
              }
            }
          }
          // the barrier orders every thread's stores before the release below (cumulative at GPU scope)
          ok = !group_bar_or<2>(fail);
          if (ok && tid == 0) {
            red_release_gpu_add(p.done, 1u);
            MEGA_STAMP(ph * 6 + 5);
          }
        }
        if (ph == 0 && tid == 0) st_release_cta(&sh->xa_free, (unsigned int)(l + 1));
      }
    }
    if (!ok && tid == 0) report_status(p.status, kStatusBarrierTimeout);  // the first code stays
  } else {
    // ================= attention warps =================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 240;");
    const int aw = warp - 8;
    const int tid = threadIdx.x - 256;
    bool fail = false, ok = true;
    for (int l = 0; l < p.L && ok; ++l) {
      const unsigned int qkv_done = (unsigned int)l * p.per_layer + (unsigned int)(p.ph[0].n_groups * p.ph[0].S);
      // The K/V blocks are staged in the activation ring: this CTA's products have read all that was in it, and it is not
      // filled again before xa_bar.
      if (!wait_seen(&sh->xa_free, (unsigned int)(l + 1), p.status)) {
        report_status(p.status, kStatusBarrierTimeout);
        fail = true;
      }
      for (int it = cta; it < p.att_items && ok; it += G) {
        const int split = it % p.splits;
        const int rest = it / p.splits;
        const int kvh = rest % p.Hkv, b = rest / p.Hkv;
        if (p.seq_lens[b] > 0) {
          if (!mega_attention_item(p.att, (long long)l * p.cache_layer_stride, split, kvh, b, xa, aw, tid, &sh->seen, qkv_done,
                                   cta == 0 && l == p.trace_layer ? p.trace : nullptr))
            fail = true;
        } else if (!wait_seen(&sh->seen, qkv_done, p.status)) {
          // an idle row (a free slot inside the batch), whose output is never used: it still counts after the qkv phase only
          report_status(p.status, kStatusPeerFlagTimeout);
          fail = true;
        }
        ok = !group_bar_or<1>(fail);  // every thread's output stores are issued, the staging area is free
        if (ok && tid == 0) red_release_gpu_add(p.done, 1u);
      }
      if (!ok) break;
      fence_proxy_async_smem();   // the activation ring is handed back to TMA
      mbar_arrive(&sh->xa_bar);
      if (tid == 0) MEGA_STAMP(25);
      if (tid == 0) MEGA_STAMP_ALL(1);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// 3-D map over per-layer weight matrices that sit at a constant stride in one flat buffer:
// (K inner, rows, layer); box = 64 x box_rows x 1, 128-byte swizzle.
CUtensorMap make_tmap_w3d(const void* base, uint64_t K, uint64_t rows, uint64_t layers, uint64_t layer_stride_elems,
                          uint32_t box_rows) {
  if ((reinterpret_cast<uint64_t>(base) & 15) != 0 || (K * 2) % 16 != 0 || (layer_stride_elems * 2) % 16 != 0)
    throw std::runtime_error("decode_layers: weight tensor map alignment");
  CUtensorMap m;
  cuuint64_t dims[3] = {K, rows, layers};
  cuuint64_t strides[2] = {K * 2, layer_stride_elems * 2};
  cuuint32_t box[3] = {kMBK, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = get_encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("decode_layers: cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return m;
}

template <int BT>
void launch_mega(const CUtensorMap* tm, const MegaParams& p, cudaStream_t stream) {
  using Cfg = MegaCfg<BT>;
  auto kernel = decode_layers_kernel<BT>;
  AGRPO_SET_MAX_DYN_SMEM(kernel, Cfg::kSmem, "decode_layers smem attr");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.grid, 1, 1);
  cfg.blockDim = dim3(kMegaThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // all CTAs resident together: they wait on one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  check_cuda(cudaLaunchKernelEx(&cfg, kernel, tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], tm[6], tm[7], p), "decode_layers launch");
}

int split_for(int n_groups, int num_kb, int grid) {
  int S = grid / n_groups;
  if (S < 1) S = 1;
  if (S > num_kb) S = num_kb;
  if (S > 16) S = 16;
  return S;
}

}  // namespace

// Bytes of fp32 scratch the kernel needs for `rows` batch rows (partial tiles of the phase with the most work items).
long long decode_layers_scratch_bytes(int rows, int H, int Q, int QD, int F, int num_sms) {
  const int BT = rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 256;
  const int groups[4] = {Q / kFT, H / kFT, F / 64, H / kFT};
  const int kbs[4] = {H / kMBK, QD / kMBK, H / kMBK, F / kMBK};
  long long items = 0;
  for (int i = 0; i < 4; ++i) {
    const long long n = (long long)groups[i] * split_for(groups[i], kbs[i], num_sms);
    if (n > items) items = n;
  }
  return items * BT * kFT * 4;
}

bool decode_layers_supported(int rows, int H, int Q, int QD, int F, int Hq, int Hkv, int head_dim) {
  return rows >= 1 && rows <= 256 && head_dim == 128 && H % 128 == 0 && Q % 128 == 0 && QD % 64 == 0 && F % 64 == 0 &&
         Q == (Hq + 2 * Hkv) * 128 && QD == Hq * 128 && Hkv > 0 && Hq % Hkv == 0 && Hq / Hkv <= 8 && Q / 128 <= 512 &&
         F / 64 <= 512 && H / 128 <= 512;
}

void launch_decode_layers(const DecodeLayersArgs& a, cudaStream_t stream) {
  if (!decode_layers_supported(a.B, a.H, a.Q, a.QD, a.F, a.Hq, a.Hkv, 128)) throw std::runtime_error("decode_layers: shape not served");
  MegaParams p;
  p.L = a.L; p.B = a.B; p.H = a.H; p.Q = a.Q; p.QD = a.QD; p.F = a.F; p.Hq = a.Hq; p.Hkv = a.Hkv;
  p.grid = a.num_sms;
  const int groups[4] = {a.Q / kFT, a.H / kFT, a.F / 64, a.H / kFT};
  const int kbs[4] = {a.H / kMBK, a.QD / kMBK, a.H / kMBK, a.F / kMBK};
  unsigned int per_layer = 0;
  long long max_items = 0;
  for (int i = 0; i < 4; ++i) {
    p.ph[i].n_groups = groups[i];
    p.ph[i].num_kb = kbs[i];
    p.ph[i].S = split_for(groups[i], kbs[i], p.grid);
    per_layer += (unsigned int)(groups[i] * p.ph[i].S);
    if ((long long)groups[i] * p.ph[i].S > max_items) max_items = (long long)groups[i] * p.ph[i].S;
  }
  p.splits = a.splits < 1 ? 1 : a.splits;
  p.att_items = a.B * a.Hkv * p.splits;
  p.per_layer = per_layer + (unsigned int)p.att_items;
  const int BT = a.B <= 32 ? 32 : a.B <= 64 ? 64 : a.B <= 128 ? 128 : 256;
  if (max_items * BT * kFT * 4 > a.partials_bytes) throw std::runtime_error("decode_layers: scratch buffer too small");
  p.x = (__nv_bfloat16*)a.x; p.x1 = (__nv_bfloat16*)a.x1; p.qkv = (__nv_bfloat16*)a.qkv; p.attn = (__nv_bfloat16*)a.attn;
  p.act = (__nv_bfloat16*)a.act;
  p.bqkv = (const __nv_bfloat16*)a.bqkv; p.bqkv_stride = a.bqkv_stride;
  p.ss = a.ss; p.ss_stride = a.ss_stride;
  p.eps = a.eps; p.inv_h = 1.f / (float)a.H;
  p.cos_t = a.cos_t; p.sin_t = a.sin_t; p.max_pos = a.max_pos;
  p.block_tables = a.block_tables; p.max_blocks = a.max_blocks; p.seq_lens = a.seq_lens;
  p.cache = (__nv_bfloat16*)a.cache; p.cache_layer_stride = a.cache_layer_stride; p.cache_v_off = a.cache_v_off;
  p.num_cache_blocks = a.num_cache_blocks;
  DecodeParams& d = p.att;
  d.q = p.qkv; d.ldq = a.Q; d.q_col0 = 0;
  d.k_cache = p.cache; d.v_cache = p.cache + a.cache_v_off;
  d.block_tables = a.block_tables; d.max_blocks = a.max_blocks; d.seq_lens = a.seq_lens; d.num_cache_blocks = a.num_cache_blocks;
  d.Hq = a.Hq; d.Hkv = a.Hkv; d.G = a.Hq / a.Hkv; d.splits = p.splits;
  d.scale_log2 = a.softmax_scale * 1.4426950408889634f;
  d.out = p.attn; d.ldo = a.QD;
  d.part_o = a.part_o; d.part_ml = a.part_ml; d.tickets = nullptr;
  p.partials = a.partials;
  p.done = a.counters;
  // A wait that runs out has to end the others, in every CTA: without a status word of the caller's they watch one of the launch's own.
  p.status = a.status != nullptr ? a.status : reinterpret_cast<int*>(a.counters + 1);
  d.status = p.status;
  p.trace = a.trace;
  p.trace_layer = a.trace_layer;
  p.trace_all = a.trace_words >= 32 + 4 * a.num_sms ? 1 : 0;
  // the counter starts from zero and the handed-over buffers from "not yet" in every launch (stream-ordered, also inside a
  // captured graph)
  check_cuda(cudaMemsetAsync(a.counters, 0, kCounterWords * sizeof(unsigned int), stream), "decode_layers counters");
  check_cuda(cudaMemsetAsync(a.partials, 0xff, (size_t)max_items * BT * kFT * 4, stream), "decode_layers partials");
  if (p.splits > 1) {
    check_cuda(cudaMemsetAsync(a.part_o, 0xff, (size_t)p.att_items * 8 * kDecD * 4, stream), "decode_layers attention partials");
    check_cuda(cudaMemsetAsync(a.part_ml, 0xff, (size_t)p.att_items * 8 * 2 * 4, stream), "decode_layers attention partials");
  }
  CUtensorMap tm[8];
  tm[0] = make_tmap_w3d(a.wqkv, a.H, a.Q, a.L, a.wqkv_stride, kFT);
  tm[1] = make_tmap_w3d(a.wo, a.QD, a.H, a.L, a.wo_stride, kFT);
  tm[2] = make_tmap_w3d(a.wgu, a.H, 2 * (uint64_t)a.F, a.L, a.wgu_stride, 64);
  tm[3] = make_tmap_w3d(a.wd, a.F, a.H, a.L, a.wd_stride, kFT);
  tm[4] = make_tmap_2d(a.x, a.H, a.rows_alloc, a.H, kMBK, BT);
  tm[5] = make_tmap_2d(a.attn, a.QD, a.rows_alloc, a.QD, kMBK, BT);
  tm[6] = make_tmap_2d(a.x1, a.H, a.rows_alloc, a.H, kMBK, BT);
  tm[7] = make_tmap_2d(a.act, a.F, a.rows_alloc, a.F, kMBK, BT);
  switch (BT) {
    case 32: launch_mega<32>(tm, p, stream); break;
    case 64: launch_mega<64>(tm, p, stream); break;
    case 128: launch_mega<128>(tm, p, stream); break;
    default: launch_mega<256>(tm, p, stream); break;
  }
}

int decode_layers_counter_words() { return kCounterWords; }

}  // namespace agrpo
