// Blackwell backward main kernel (head_dim 64, 16-bit): tcgen05 MMAs with every accumulator in TMEM.
// Same mathematics as bwd_mma.cu (reference: csrc/mfa_steel_bwd.cpp:284-745, 765-1293); the preprocess
// (delta, dQ accumulator reset) and the final dQ conversion are shared with it.
//
// One persistent CTA per SM takes work items from a global counter; an item is a tile of 128 keys of one kv head, for
// which the CTA walks the query heads of the GQA group and the 128-row query tiles that can see those keys.  Per query tile, five GEMMs, all M = 128:
//   S^T  = K . Q^T      (A = K rows in TMEM, per half of 64 queries, K = 64)   -> TMEM [0,64) and [128,192)
//   dP^T = V . dO^T     (A = V rows in TMEM, per half)                          -> TMEM [64,128) and [192,256)
//   and a fifth k-step each, constants against three 16-bit parts of the query's -L / (scale*log2e) or -delta
//   (Parts3): the compute warps read neither from shared memory, which was 400 of 1480 clk of a half's arithmetic (with a
//   soft cap L is subtracted after the cap, from shared memory)
//   8 compute warps (thread = key row, four warps per query half) turn these into
//   P^T = 2^(scale*log2e*S^T) and dS^T = P^T o dP^T, written back as 16-bit A operands over
//   the columns they came from, and dS^T also to shared memory as a [query block][key][64 queries] tile
//   dV  += P^T . dO     (A from TMEM, B = dO as an MN-major operand, N = 64)   -> TMEM [256,320)
//   dK  += dS^T . Q     (A from TMEM, B = Q MN-major)                          -> TMEM [320,384)
//   dQ   = dS . K       (SS: A = the dS^T tile read MN-major, B = K MN-major)  -> TMEM [384,448)
// K and V rows sit in TMEM [448,512) as A operands for the CTA's lifetime (copied there once by the compute warps),
// so S^T / dP^T read only the query tiles from shared memory.
// The two query halves have their own S^T / dP^T columns, their own compute warps, stages of Q / dO and barriers, and dS has
// two shared-memory buffers, so the MMAs of one half (and its next S^T / dP^T) run while the other half's warps compute.
// What bounds it: each half's chain (arrival, MMAs 570 clk, S^T seen, arithmetic 950 to 1130, stores), whose barriers and
// stores are slow beside the MMAs' shared-memory reads; a 128 x 128 step takes 2780 clk, of which the MMA warp issues
// during 1630 (3160 with all eight warps on both halves in turn, L and delta from shared memory and staged by the
// producer).  Sixteen compute warps (80 registers): 3140.  dQ is read out of TMEM by
// four flush warps, staged in shared memory and added to the fp32 accumulator by TMA reduce-add copies (whole 128-byte
// lines per request; per-lane red.global.add touched 32 lines per instruction and was bound by the load/store unit);
// dK / dV leave TMEM once, at the end, through shared memory as whole rows.
// Warp 8 is the TMA producer (Q, dO double-buffered), warp 14 stages L and delta, warp 9 issues the
// MMAs (the whole warp waits, one elected lane issues a group: 46 clk per N = 64 MMA became 33 to 38, and the backward of
// B=2 16/4 heads 8192^2 causal 1072 -> 950 us), warps 10-13 move dQ from TMEM to the fp32 accumulator; warp 10 also fetches the next item and starts its K / V
// loads while the current item runs.  No load uses cluster multicast; every
// mbarrier wait is bounded.
#include <type_traits>

#include "common.cuh"
#include "launch.h"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace b200fa {
// Device status word of this file's kernels: bit 0 = a bounded wait gave up.
static __device__ int g_kernel_status = 0;


namespace {

constexpr int BK = 128;      // keys per CTA (TMEM lanes)
constexpr int BQ = 128;      // queries per step
constexpr int HD = 64;
constexpr int kThreads = 480;       // warps 0-7 compute, 8 producer, 9 MMA issue, 10-13 dQ flush, 14 L and delta
constexpr int kProducerWarp = 8, kMmaWarp = 9, kFlushWarp = 10, kStatWarp = 14;
constexpr uint32_t kTmemCols = 512;
// query half x (64 queries): S^T at cST + 128x, dP^T at cDPT + 128x
constexpr uint32_t cST = 0, cDPT = 64, cDV = 256, cDK = 320, cDQ = 384;
// K and V rows as 16-bit A operands (two elements per column), written once per CTA
constexpr uint32_t cKA = 448, cVA = 480;

constexpr int kTileBytes = 128 * HD * 2;                 // 16384: one [128 rows][64] tile
constexpr int kDSBytes = BQ * BK * 2;                    // 32768: dS as two 64-key halves [half][query][128 B]
// In front of the tiles, for the k-steps that subtract L and delta: the constant A operand (128 rows x 8 values), the B operands
// of L and of delta per stage and half (64 queries x 8) and zeros, the other 8 of a k-step's 16 for all of them; then -L in
// fp32 for a soft cap, which is applied to the score before L is subtracted
constexpr int kConstBytes = BK * 16, kAugBytes = 64 * 16, kZeroBytes = BK * 16;
constexpr int kStatBytes = kConstBytes + 8 * kAugBytes + kZeroBytes + 2 * BQ * 4;
constexpr int kDQStageBytes = BQ * HD * 4;               // 32768: dQ tile in fp32, two 32-column halves [half][query][128 B]
// K, V, Q x2, dO x2, dS x2, dQ, second K buffer (the next work item's keys) = 212992
constexpr int kSmemTiles = 2 * kTileBytes + 4 * kTileBytes + 2 * kDSBytes + kDQStageBytes + kTileBytes;
constexpr int kSmemBytes = kSmemTiles + kStatBytes + 256 + 1024;
static_assert(kStatBytes % 1024 == 0 && kSmemTiles % 1024 == 0 && kSmemBytes <= 227 * 1024, "shared memory");

// BAR_KV (+ K buffer) live for the whole kernel; the others are set up again for every work item
enum Bar {
  BAR_KV = 0,
  BAR_Q_FULL = 2,        // + 2 * stage + half: Q, dO, -L and -delta of the 64 queries of a half
  BAR_Q_EMPTY = 6,       // + 2 * stage + half
  BAR_ST_DONE = 10,      // + half
  BAR_PD_READY = 12,     // + half
  BAR_DQ_DONE = 14,
  BAR_DQ_FREE = 15,
  BAR_KV_TMEM = 16,
  BAR_ACC_DONE = 17,
  BAR_COUNT = 18
};

struct BwdArgs {
  BwdParams p;
  int dtype;
  int gx, gy, total_items;      // work items: (key tile, kv head, batch | sequence)
  int group;                    // their order: item_of
  int parts;                    // PARTS: an item's (query head, query tile) steps are cut into so many items, each leaving
  float* part;                  // fp32 sums [part][dK, dV][B, Hkv, S][64], which launch_dkv_reduce adds up
  int* counter;                 // next work item (zeroed by the preprocess kernel)
};

// Not volatile: the loads may be scheduled ahead of the (volatile) dS stores of earlier elements, which hides their
// latency.  The address must come from opaque_u32() issued after the wait that makes the data visible, so that no
// load moves above that wait and none is merged with the same address of another tile.
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 v;
  asm("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void lds_v4u(uint32_t addr, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t opaque_u32(uint32_t x) {
  uint32_t y;
  asm volatile("mov.u32 %0, %1;\n" : "=r"(y) : "r"(x) : "memory");
  return y;
}
// DT: 0 = float16, 1 = bfloat16 (a template parameter so that each pair is converted once, not once per type)
template <int DT> __device__ __forceinline__ uint32_t pack16b(float a, float b) {
  return DT == 0 ? Elem<__half>::pack(a, b) : Elem<__nv_bfloat16>::pack(a, b);
}

// A float as a sum of three 16-bit values times constants (that the A operand of the k-step has): exact to 2^-24 of it or
// better.  bfloat16 has float's range.  float16 does not: its constants spread the three parts over 2^31 .. 2^-33 (dS, which is
// rounded to float16, has no bits below 2^-24).  What is larger than kMax, or not a number, becomes NaN.
template <int DT> struct Parts3 {
  static constexpr float c0 = DT == 0 ? 32768.f : 1.f, c1 = DT == 0 ? 16.f : 1.f, c2 = DT == 0 ? 1.f / 256.f : 1.f;
  static constexpr float kMax = DT == 0 ? 65504.f * 32768.f : 1.7014118e38f;
  // the parts of v as a row of the B operand
  static __device__ __forceinline__ uint4 split(float v) {
    auto round16 = [](float x) -> float { return DT == 0 ? __half2float(__float2half_rn(x)) : __bfloat162float(__float2bfloat16_rn(x)); };
    if (!(fabsf(v) <= kMax)) v = NAN;
    const float a = round16(v * (1.f / c0));
    const float r1 = v - a * c0, b = round16(r1 * (1.f / c1));
    const float r2 = r1 - b * c1, c = round16(r2 * (1.f / c2));
    return make_uint4(pack16b<DT>(a, b), pack16b<DT>(c, 0.f), 0u, 0u);
  }
};

// CAP: the forward capped the scores (cap * tanh(s / cap)); P is rebuilt from the capped score and dS carries the
// factor 1 - tanh^2.  WIN: a left window (fewer query tiles per key tile, one more test in the masked tiles).  Both are
// compile-time variants, so that the plain kernel's loops are untouched (with the window test compiled into every
// instance config 5's backward ran 9 % slower).
// FEAT: the ALiBi bias slope[h] * (key - (query + S - N)) and / or a block mask (cells of mask_bq x mask_bk, mask_bq a
// multiple of 32 so that the 32 queries a thread handles per step share one cell), as the forward's feature
// instantiation applies them (csrc/mfa_steel_fwd.cpp:951-970, 230-262 in the reference).  Without CAP / WIN.
// PARTS: items are cut (a.parts > 1); a variant of its own, because these kernels slow down with every register more.
template <int DT, bool CAP, bool WIN, bool FEAT, bool PARTS>
__global__ void __launch_bounds__(kThreads, 1)
bwd_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                 const __grid_constant__ CUtensorMap tmDQ, const BwdArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sConst = smem;                        // [128][16 B]: the parts' constants in every row
  unsigned char* sAug = sConst + kConstBytes;          // [2 stages][2 halves][64][16 B]: parts of -L / scale_log2; the same of -delta
  unsigned char* sZero = sAug + 8 * kAugBytes;
  float* sL = reinterpret_cast<float*>(sZero + kZeroBytes);    // [2][BQ], soft cap only
  unsigned char* sK = smem + kStatBytes;
  unsigned char* sV = sK + kTileBytes;
  unsigned char* sQ = sV + kTileBytes;                 // [2][128][128 B]
  unsigned char* sDO = sQ + 2 * kTileBytes;            // [2][128][128 B]
  unsigned char* sDS = sDO + 2 * kTileBytes;           // [2 buffers][2 key halves][128 queries][128 B]
  unsigned char* sDQ = sDS + 2 * kDSBytes;             // [2 column halves][128 queries][128 B] fp32, 128B-swizzled
  unsigned char* sK1 = sDQ + kDQStageBytes;            // K of every other work item
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSmemTiles + kStatBytes);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + BAR_COUNT);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  // [2][8]: this item and the next one as {index or -1, key tile, kv head, batch, k_begin, S, q_begin, N}
  volatile int* s_work = reinterpret_cast<volatile int*>(s_tmem + 2);

  const BwdParams& p = a.p;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar = [&](int i) -> uint32_t { return smem_u32(&bars[i]); };

  // Persistent CTA, one per SM: work items (128 keys of one kv head of one batch entry or sequence) come from a global
  // counter in the order of item_of, a group of heads' key tiles with the most query tiles first.  While an item runs,
  // the producer thread fetches the next one and starts its K load (second buffer) and, once this item's V sits
  // in TMEM, its V load; set-up, K/V latency and the gap between CTAs are paid once per SM instead of once per item.
  // Next item that has keys (grid cells beyond a sequence's end are skipped), decoded into slot `sl` of s_work for
  // every role to read; index -1 when the list is exhausted.  Run by one thread, with global latency per try.
  auto fetch_next = [&](int sl) -> int {
    volatile int* o = s_work + sl * 8;
    for (int tries = 0; tries < (1 << 24); ++tries) {
      const int idx = atomicAdd(a.counter, 1);
      if (idx >= a.total_items) break;
      int kt, pair;
      item_of(idx, a.gx, a.total_items / a.gx, a.group, kt, pair);
      const int part_ = PARTS ? pair % a.parts : 0;
      if constexpr (PARTS) pair /= a.parts;
      const int kvh_ = pair % a.gy, z = pair / a.gy;
      int kb = 0, S_ = p.S, qb = 0, N_ = p.N;
      if (p.cu_k != nullptr) {
        kb = p.cu_k[z];
        S_ = p.cu_k[z + 1] - kb;
      }
      if (kt * BK >= S_) continue;
      if (p.cu_q != nullptr) {
        qb = p.cu_q[z];
        N_ = p.cu_q[z + 1] - qb;
      }
      o[1] = kt | (part_ << 24); o[2] = kvh_; o[3] = p.cu_q != nullptr ? 0 : z; o[4] = kb; o[5] = S_; o[6] = qb; o[7] = N_;
      o[0] = idx;
      return idx;
    }
    o[0] = -1;
    return -1;
  };
  // K / V tile of the item in slot `sl`
  auto load_k_of = [&](int sl, unsigned char* dst, uint32_t b) {
    volatile int* o = s_work + sl * 8;
    tma_load_4d(smem_u32(dst), &tmK, b, 0, o[4] + (o[1] & 0xffffff) * BK, o[2], o[3]);
  };
  auto load_v_of = [&](int sl, uint32_t b) {
    volatile int* o = s_work + sl * 8;
    tma_load_4d(smem_u32(sV), &tmV, b, 0, o[4] + (o[1] & 0xffffff) * BK, o[2], o[3]);
  };
  if (warp == kProducerWarp && lane == 0) {
    mbar_init(bar(BAR_KV), 1);
    mbar_init(bar(BAR_KV + 1), 1);
    *s_abort = 0;
    fence_barrier_init();
    fence_proxy_async();
    if (fetch_next(0) >= 0) {
      mbar_arrive_expect_tx(bar(BAR_KV), 2 * kTileBytes);
      load_k_of(0, sK, bar(BAR_KV));
      load_v_of(0, bar(BAR_KV));
    }
  }
  {
    // the k-step that subtracts L and delta: S^T -= L / scale_log2, dP^T -= delta, each query's value in every key row
    using P3 = Parts3<DT>;
    for (int i = tid; i < 2 * BK; i += kThreads)
      *reinterpret_cast<uint4*>(i < BK ? sConst + i * 16 : sZero + (i - BK) * 16) =
          i < BK ? make_uint4(pack16b<DT>(P3::c0, P3::c1), pack16b<DT>(P3::c2, 0.f), 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(s_tmem), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;

  for (int w = 0;; ++w) {
  volatile int* wk = s_work + (w & 1) * 8;
  if (wk[0] < 0 || *s_abort != 0) break;
  const int kvh = wk[2], bb = wk[3], k_begin = wk[4], S = wk[5], q_begin = wk[6], N = wk[7];
  const int n0 = (wk[1] & 0xffffff) * BK;
  const int off = S - N;
  int m_begin = 0;
  if (p.causal) m_begin = max(0, n0 - off) / BQ;
  int m_end = (N + BQ - 1) / BQ;
  // a left window: the last row that still sees this tile's last key is i = key - off + window_left
  if constexpr (WIN) m_end = min(m_end, max(0, min(S, n0 + BK) - 1 - off + p.window_left) / BQ + 1);
  const int nm = max(0, m_end - m_begin);
  // this item's steps of (query head, query tile): it0 + it
  const int it0 = PARTS ? nm * p.gqa * (wk[1] >> 24) / a.parts : 0;
  const int nm_or_1 = max(nm, 1);
  const int n_iter = PARTS ? nm * p.gqa * ((wk[1] >> 24) + 1) / a.parts - it0 : nm * p.gqa;
  const int kbuf = w & 1;                              // K buffer and KV barrier of this item
  const uint32_t kv_par = (w >> 1) & 1;
  unsigned char* sKc = kbuf ? sK1 : sK;

  // The producer thread sets up this item's barriers and starts the loads of its first two Q / dO tiles (all stages
  // are empty) before the CTA-wide sync.
  // a half of a tile at a time: its stage is free again as soon as the half's own dV and dK have read it
  auto load_q = [&](int it, int x, int m, int hq) {
    const int st = it & 1, row = q_begin + m * BQ + 64 * x;
    const uint32_t b = bar(BAR_Q_FULL + 2 * st + x);
    mbar_arrive_expect_tx(b, kTileBytes);
    tma_load_4d(smem_u32(sQ + st * kTileBytes + x * (kTileBytes / 2)), &tmQ, b, 0, row, hq, bb);
    tma_load_4d(smem_u32(sDO + st * kTileBytes + x * (kTileBytes / 2)), &tmDO, b, 0, row, hq, bb);
  };
  if (warp == kProducerWarp && lane == 0) {
    if (w > 0)
      for (int i = BAR_Q_FULL; i < BAR_COUNT; ++i) mbar_inval(bar(i));    // nobody waits or arrives between items
    for (int s = 0; s < 4; ++s) {
      mbar_init(bar(BAR_Q_FULL + s), 2);    // the loads' bytes and the warp that stages L and delta
      mbar_init(bar(BAR_Q_EMPTY + s), 1);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(bar(BAR_ST_DONE + x), 1);
      mbar_init(bar(BAR_PD_READY + x), 4);  // one arrive per compute warp of the half
    }
    mbar_init(bar(BAR_DQ_DONE), 1);
    mbar_init(bar(BAR_ACC_DONE), 1);
    mbar_init(bar(BAR_DQ_FREE), 4);       // one arrive per flush warp
    mbar_init(bar(BAR_KV_TMEM), 8);       // one arrive per warp that copies K or V there
    fence_barrier_init();
    fence_proxy_async();
    for (int it = 0; it < 2 && it < n_iter; ++it)
      for (int x = 0; x < 2; ++x) load_q(it, x, m_begin + (it0 + it) % nm, kvh * p.gqa + (it0 + it) / nm);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == kProducerWarp) {
    // ============================ producer ============================
    if (lane == 0) {
      int r_it = (it0 + 2) % nm_or_1, hq_it = kvh * p.gqa + (it0 + 2) / nm_or_1;
      for (int u = 4; u < 2 * n_iter; ++u) {
        const int it = u >> 1, x = u & 1;
        if (!mbar_wait_bounded(bar(BAR_Q_EMPTY + 2 * (it & 1) + x), ((it >> 1) & 1) ^ 1, s_abort)) break;
        load_q(it, x, m_begin + r_it, hq_it);
        if (x == 1 && ++r_it == nm) { r_it = 0; ++hq_it; }
      }
    }
  } else if (warp == kStatWarp) {
    // ============================ L and delta ============================
    // of a half's 64 query rows, into the stage that its Q rows go to.  They are loaded a unit (half tile) ahead, and by a
    // warp of their own: in the producer's, their latency and arithmetic (620 clk a unit) held up its Q / dO loads.
    // Rows beyond N, or without any visible key, get an L that makes their P exactly zero.
    float Ln[2], dn[2];
    int r_l = it0 % nm_or_1, hq_l = kvh * p.gqa + it0 / nm_or_1;       // tile of the next L / delta load
    auto load_stat = [&](int u) {
      const int row0 = (m_begin + r_l) * BQ + (u & 1) * 64 + lane * 2;
      const int64_t idx = bb * p.lse_bs + hq_l * p.lse_hs + q_begin + row0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const bool in = row0 + i < N;
        Ln[i] = in ? p.lse[idx + i] : -INFINITY;
        dn[i] = in ? p.delta[idx + i] : 0.f;
      }
      if ((u & 1) && ++r_l == nm) { r_l = 0; ++hq_l; }
    };
    const float inv_scale = 1.f / p.scale_log2;
    if (n_iter > 0) load_stat(0);
    for (int u = 0; u < 2 * n_iter; ++u) {
      const int it = u >> 1, x = u & 1, st = it & 1;
      if (it >= 2 && !__all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_Q_EMPTY + 2 * st + x), ((it >> 1) & 1) ^ 1, s_abort))) break;
      const float L0 = Ln[0], L1 = Ln[1], d0 = dn[0], d1 = dn[1];
      if (u + 1 < 2 * n_iter) load_stat(u + 1);
      // A row that sees no key, or is not there, gets the largest value: its P is zero
      auto l_part = [&](float L) { return Parts3<DT>::split(fabsf(L) == INFINITY ? -copysignf(Parts3<DT>::kMax, inv_scale) : -L * inv_scale); };
      if constexpr (CAP) {
        // stored negated: the compute loop adds it
        *reinterpret_cast<float2*>(sL + st * BQ + x * 64 + lane * 2) = make_float2(L0 == -INFINITY ? -INFINITY : -L0, L1 == -INFINITY ? -INFINITY : -L1);
      }
      // L and delta have operands of their own: a delta that is not finite makes its query's dP^T NaN and leaves S^T, and so dV,
      // alone (0 x NaN is NaN, so a shared row of parts would not)
      uint4* t = reinterpret_cast<uint4*>(sAug + (2 * st + x) * kAugBytes) + lane * 2;
      if constexpr (!CAP) {
        t[0] = l_part(L0);
        t[1] = l_part(L1);
      }
      t += 4 * kAugBytes / 16;
      t[0] = Parts3<DT>::split(-d0);
      t[1] = Parts3<DT>::split(-d1);
      fence_proxy_async();           // written with ordinary stores, read by the MMAs
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(BAR_Q_FULL + 2 * st + x));
      __syncwarp();
    }
  } else if (warp == kMmaWarp) {
   if (n_iter > 0) {
    // ============================ MMA issue ============================
    // Per query tile t and query half x: [S^T_x, dP^T_x] -> (compute) -> [dV += P^T_x.dO_x, dK += dS^T_x.Q_x]; after both
    // halves dQ = dS.K.  Issue order keeps the pipe fed while the compute warps work on the other half:
    //   ST/DPT a,b (t=0) | PD_a -> dV_a dK_a, ST/DPT a (t+1) | PD_b -> dV_b dK_b, dQ, ST/DPT b (t+1) | ...
    // The whole warp waits, one elected lane issues a group of MMAs (see elect_one).
    auto wait = [&](int i, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait_bounded(bar(i), parity, s_abort)); };
    const uint32_t id_st = instr_desc(DT, 0, 128, 64);     // S^T, dP^T of one half: B K-major, N = 64
    const uint32_t id_mn = instr_desc(DT, 1, 128, HD);     // dV, dK: B MN-major, N = 64
    const uint32_t id_dq = id_mn | (1u << 15);             // dQ: A (dS^T as stored) MN-major as well
    const uint64_t kmn = smem_desc(smem_u32(sKc), kTileBytes, 1024);
    // dS^T [query block of 64][key][128 B]: MN (query) blocks kTileBytes apart, 8-key groups 1024 apart
    const uint64_t dsd0 = smem_desc(smem_u32(sDS), kTileBytes, 1024);
    const uint64_t qd0 = smem_desc(smem_u32(sQ), 16, 1024), dod0 = smem_desc(smem_u32(sDO), 16, 1024);
    const uint64_t qmn0 = smem_desc(smem_u32(sQ), kTileBytes, 1024), domn0 = smem_desc(smem_u32(sDO), kTileBytes, 1024);
    const uint64_t constd = smem_desc_plain(smem_u32(sConst), static_cast<uint32_t>(sZero - sConst), 128);
    const uint64_t augd0 = smem_desc_plain(smem_u32(sAug), static_cast<uint32_t>(sZero - sAug), 128);
    constexpr uint64_t kAugU = (kAugBytes >> 4) - (static_cast<uint64_t>(kAugBytes >> 4) << 16);     // the next one, as much nearer to the zeros
    constexpr uint64_t kTileU = kTileBytes >> 4, kHalfRowsU = (64 * 128) >> 4, kDSU = kDSBytes >> 4;
    bool ok = wait(BAR_KV_TMEM, 0);
    tc_fence_after();
    // S^T_x and dP^T_x of tile `it`: A = K / V rows in TMEM (8 columns per 16 head-dim elements), B rows = the 64
    // queries of half x
    // Each tcgen05.mma waits for room in a queue about one MMA deep (in a microbenchmark the issue loop ends as the
    // last MMA completes), so whatever else this warp does is a bubble in the tensor pipe.  It therefore waits on
    // two barriers per tile only (PD_READY of each half): the compute warps check, before they arrive there, that the
    // next tile's Q / dO have landed (half a) and that the flush warps have read the previous dQ (half b).
    auto issue_stdp = [&](int it, int x) {
      const int st = it & 1;
      const uint64_t qd = qd0 + st * kTileU + x * kHalfRowsU, dod = dod0 + st * kTileU + x * kHalfRowsU;
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        mma_ts(tmem + cST + 128 * x, tmem + cKA + k * 8, qd + k * 2, id_st, k > 0 ? 1u : 0u);
      const uint64_t aug = augd0 + (2 * st + x) * kAugU;
      if constexpr (!CAP) mma_ss(tmem + cST + 128 * x, constd, aug, id_st, 1u);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        mma_ts(tmem + cDPT + 128 * x, tmem + cVA + k * 8, dod + k * 2, id_st, k > 0 ? 1u : 0u);
      mma_ss(tmem + cDPT + 128 * x, constd, aug + 4 * kAugU, id_st, 1u);
      tc_commit(bar(BAR_ST_DONE + x));
    };
    for (int x = 0; x < 2 && ok; ++x) {
      ok = wait(BAR_Q_FULL + x, 0);
      if (ok && elect_one()) issue_stdp(0, x);
      __syncwarp();
    }
    for (int it = 0; it < n_iter && ok; ++it) {
      const int st = it & 1;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        if (!wait(BAR_PD_READY + x, it & 1)) { ok = false; break; }
        tc_fence_after();
        const uint64_t qmn = qmn0 + st * kTileU + x * kHalfRowsU, domn = domn0 + st * kTileU + x * kHalfRowsU;
        // A in TMEM: 8 columns per 16 queries; queries 0-31 of the half at +0, 32-63 at +32 (each part over the scores
        // it was made from); B rows = queries, 16 rows = 128 units
        if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_ts(tmem + cDV, tmem + cST + 128 * x + (k >> 1) * 32 + (k & 1) * 8, domn + k * 128, id_mn,
                             (it > 0 || x > 0 || k > 0) ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_ts(tmem + cDK, tmem + cDPT + 128 * x + (k >> 1) * 32 + (k & 1) * 8, qmn + k * 128, id_mn,
                             (it > 0 || x > 0 || k > 0) ? 1u : 0u);
        // the buffers of half x are free again (the MMAs above read them in pipe order before anything issued now); half b's
        // next scores go before dQ, which nobody waits for as soon
        tc_commit(bar(BAR_Q_EMPTY + 2 * st + x));
        if (it + 1 < n_iter) issue_stdp(it + 1, x);
        if (x == 1) {
          // dQ = dS.K: A = dS^T rows = keys (buffer it & 1), B = K rows = keys, 16 keys = 128 units per step; the
          // flush warps have read the previous tile's dQ out of TMEM (the compute warps saw DQ_FREE before PD_READY)
          const uint64_t dsd = dsd0 + (it & 1) * kDSU;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            mma_ss(tmem + cDQ, dsd + k * 128, kmn + k * 128, id_dq, k > 0 ? 1u : 0u);
          tc_commit(bar(BAR_DQ_DONE));
          if (it + 1 == n_iter) tc_commit(bar(BAR_ACC_DONE));
        }
        }
        __syncwarp();
      }
    }
   }
  } else if (warp >= kFlushWarp) {
    // ============================ dQ flush warps 10-13 ============================
    // dQ of each tile leaves TMEM here (rows = queries), is staged in shared memory in the tensor map's 128B-swizzled
    // layout and added to the fp32 accumulator by two TMA reduce-add copies per warp (32 rows x 32 columns each), off
    // the compute warps' critical path.  TMEM is handed back as soon as the tile is in registers.
    const int wq = warp & 3;                                  // TMEM lane quarter this warp may touch
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t stage = smem_u32(sDQ) + wq * 4096;         // this warp's 32 rows; the other column half is 16384 on
    const uint32_t row_addr = stage + lane * 128;
    if (warp == kFlushWarp) {
      // This warp has the most slack at the start of an item (the first dQ is thousands of clocks away): it fetches the
      // item after this one, starts its K load into the other K buffer and, when this item's V has been copied to
      // TMEM (or, for an item without query tiles, has landed), its V load.
      int nxt = -1;
      if (lane == 0) {
        nxt = fetch_next((w + 1) & 1);
        if (nxt >= 0) {
          mbar_arrive_expect_tx(bar(BAR_KV + (kbuf ^ 1)), 2 * kTileBytes);
          load_k_of((w + 1) & 1, kbuf ? sK : sK1, bar(BAR_KV + (kbuf ^ 1)));
        }
      }
      nxt = __shfl_sync(0xffffffffu, nxt, 0);
      if (nxt >= 0 || n_iter == 0) {          // without query tiles nobody else waits for this item's copies to land
        const bool pass = n_iter > 0 ? mbar_wait_bounded(bar(BAR_KV_TMEM), 0, s_abort)
                                     : mbar_wait_bounded(bar(BAR_KV + kbuf), kv_par, s_abort);
        if (__all_sync(0xffffffffu, pass) && nxt >= 0 && lane == 0) load_v_of((w + 1) & 1, bar(BAR_KV + (kbuf ^ 1)));
      }
    }
    int r_it = it0 % nm_or_1, hq_it = kvh * p.gqa + it0 / nm_or_1;    // query tile and head of this step
    for (int it = 0; it < n_iter; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_DQ_DONE), it & 1, s_abort))) break;
      tc_fence_after();
      const int hq = hq_it, m = m_begin + r_it;
      if (++r_it == nm) { r_it = 0; ++hq_it; }
      uint32_t r0[32], r1[32];
      tmem_ld32(tmem + lane_base + cDQ, r0);
      tmem_ld32(tmem + lane_base + cDQ + 32, r1);
      tc_wait_ld();
      // everything is in registers: the MMA warp may overwrite dQ
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar(BAR_DQ_FREE));
        tma_store_wait_read<0>();                             // the previous tile's copies have read the staging rows
      }
      __syncwarp();
      // rows of this group beyond the sequence hold exact zeros (their P is zero): nothing to add
      if (m * BQ + wq * 32 < N) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t o = static_cast<uint32_t>((c ^ (lane & 7)) << 4);
          sts_v4(row_addr + o, r0[4 * c], r0[4 * c + 1], r0[4 * c + 2], r0[4 * c + 3]);
          sts_v4(row_addr + 16384 + o, r1[4 * c], r1[4 * c + 1], r1[4 * c + 2], r1[4 * c + 3]);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          const int row0 = q_begin + m * BQ + wq * 32;
          tma_reduce_add_4d(&tmDQ, stage, 0, row0, hq, bb);
          tma_reduce_add_4d(&tmDQ, stage + 16384, 32, row0, hq, bb);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_read<0>();   // the copies have left shared memory; the kernel's end makes them visible
  } else {
    // ============================ compute warps 0-7 ============================
    // four warps per query half x, so that a half's waits and TMEM latency pass under the other half's arithmetic
    const int wq = warp & 3, x = warp >> 2;                  // TMEM lane quarter, query half
    const int rloc = wq * 32 + lane;                         // key row (S^T, dK, dV) or query row (dQ) inside the tile
    const int key = n0 + rloc;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    auto part_row = [&](int which, int k) -> float* {
      return a.part + ((static_cast<int64_t>((wk[1] >> 24) * 2 + which) * p.B + bb) * p.Hkv + kvh) * p.S * HD + static_cast<int64_t>(k) * HD;
    };
    if (n_iter == 0) {
      // no query sees these keys (or this part has no step): dK = dV = 0
      if (PARTS && key < S) {
        float4* pt = reinterpret_cast<float4*>(part_row(x, key));
#pragma unroll
        for (int i = 0; i < 16; ++i) pt[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else if (key < S) {
        const int64_t o = bb * p.dk_bs + kvh * p.dk_hs + static_cast<int64_t>(k_begin + key) * p.dk_rs;
#pragma unroll
        for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(x == 0 ? p.dk : p.dv) + o)[i] = make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
    bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_KV + kbuf), kv_par, s_abort));
    if (ok) {
      // K rows (warps 0-3) and V rows (warps 4-7) go to TMEM once, as the A operands of S^T and dP^T: their MMAs then
      // read only the query tiles from shared memory, whose bandwidth is what bounds this kernel
      const uint32_t rowa = smem_u32(x == 0 ? sKc : sV) + rloc * 128;
      uint32_t kr[32];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        lds_v4u(rowa + static_cast<uint32_t>((c ^ (rloc & 7)) << 4), kr[4 * c], kr[4 * c + 1], kr[4 * c + 2], kr[4 * c + 3]);
      tmem_st32(tmem + lane_base + (x == 0 ? cKA : cVA), kr);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(BAR_KV_TMEM));
    }

    int r_it = it0 % nm, hq_it = kvh * p.gqa + it0 / nm;      // query tile and head of this step
    for (int it = 0; it < n_iter && ok; ++it) {
      const int st = it & 1;
      const int m = m_begin + r_it;
      // this tile's Q, L and delta: seen before the last tile's arrival at PD_READY
      if (it == 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_Q_FULL + x), 0, s_abort))) { ok = false; break; }
      [[maybe_unused]] const uint32_t Ls = opaque_u32(smem_u32(sL + st * BQ));
      const bool need_mask = (n0 + BK > S) || (p.causal && (n0 + BK - 1 > m * BQ + off)) ||
                             (WIN && (n0 < m * BQ + BQ - 1 + off - p.window_left));
      const int wlo = WIN ? off - p.window_left : 0;    // window: key visible iff key >= qrow + wlo
      // dS^T[this key][query] lives in buffer it & 1 as [query block of 64][key][128 B], 16-byte chunks swizzled by
      // key & 7: each thread stores its 32 queries as four 16-byte chunks
      const uint32_t ds_row = smem_u32(sDS) + (it & 1) * kDSBytes + rloc * 128;
      const float2 c2 = make_float2(p.scale_log2, p.scale_log2);
      const float alibi_l2 = (FEAT && p.alibi != nullptr) ? p.alibi[hq_it] * kLog2e : 0.f;
      const float cap_in = CAP ? p.scale / p.softcap : 0.f, cap_out = p.softcap * kLog2e;
      const bool precise_tanh = p.softcap >= kPreciseTanhMinCap;

      // 32 of the half's 64 queries
      auto run_part = [&](int hf, auto masked) {
        const int q0l = x * 64 + hf * 32;                  // first of them inside the tile
        // FEAT: the mask cell of (these 32 queries, this key) and the bias of the first of them, in the log2 domain
        [[maybe_unused]] bool cell_on = true;
        [[maybe_unused]] float ab = 0.f;
        if constexpr (FEAT) {
          const int qrow0 = m * BQ + q0l;
          if (p.bmask != nullptr)
            cell_on = key < S && p.bmask[static_cast<int64_t>(min(qrow0, N - 1) / p.bm_bq) * p.bm_nk + key / p.bm_bk] != 0;
          ab = alibi_l2 * static_cast<float>(key - off - qrow0);
        }
        uint32_t rs[32], rd[32];
        tmem_ld32(tmem + lane_base + cST + 128 * x + hf * 32, rs);
        tmem_ld32(tmem + lane_base + cDPT + 128 * x + hf * 32, rd);
        tc_wait_ld();
        uint32_t pp[16], pd[16];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          [[maybe_unused]] float4 nL;
          if constexpr (CAP) {
            nL = lds_f4(Ls + (q0l + i) * 4);                 // -L of four queries
          }
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 sv = make_float2(__uint_as_float(rs[i + e]), __uint_as_float(rs[i + e + 1]));
            const float2 dv = make_float2(__uint_as_float(rd[i + e]), __uint_as_float(rd[i + e + 1]));
            float2 t;
            [[maybe_unused]] float2 dcap;
            if constexpr (CAP) {
              const float2 th = make_float2(cap_tanh(sv.x * cap_in, precise_tanh), cap_tanh(sv.y * cap_in, precise_tanh));
              t = __ffma2_rn(th, make_float2(cap_out, cap_out), e == 0 ? make_float2(nL.x, nL.y) : make_float2(nL.z, nL.w));
              dcap = __ffma2_rn(make_float2(-th.x, -th.y), th, make_float2(1.f, 1.f));
            } else {
              t = __fmul2_rn(sv, c2);                      // L is in S^T, delta in dP^T
            }
            if constexpr (FEAT) {
              t = __fadd2_rn(t, make_float2(fmaf(-alibi_l2, static_cast<float>(i + e), ab), fmaf(-alibi_l2, static_cast<float>(i + e + 1), ab)));
            }
            float2 pe = make_float2(fast_exp2(t.x), fast_exp2(t.y));
            if constexpr (FEAT) {
              if (!cell_on) pe = make_float2(0.f, 0.f);
            }
            if constexpr (decltype(masked)::value) {
              const int qrow = m * BQ + q0l + i + e;
              const bool kin = key < S;
              if (!(kin && (!p.causal || key <= qrow + off) && (!WIN || key >= qrow + wlo))) pe.x = 0.f;
              if (!(kin && (!p.causal || key <= qrow + 1 + off) && (!WIN || key >= qrow + 1 + wlo))) pe.y = 0.f;
            }
            float2 dsv;
            if constexpr (CAP) dsv = __fmul2_rn(__fmul2_rn(pe, dv), dcap);
            else dsv = __fmul2_rn(pe, dv);
            pp[(i + e) >> 1] = pack16b<DT>(pe.x, pe.y);
            pd[(i + e) >> 1] = pack16b<DT>(dsv.x, dsv.y);
          }
        }
        // P^T and dS^T go back as 16-bit pairs along the query index, inside the 32 columns this warp has just read
        // (it reads the half's other 32 after these)
        tmem_st16(tmem + lane_base + cST + 128 * x + hf * 32, pp);
        tmem_st16(tmem + lane_base + cDPT + 128 * x + hf * 32, pd);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          sts_v4(ds_row + x * kTileBytes + static_cast<uint32_t>(((hf * 4 + j) ^ (rloc & 7)) << 4), pd[4 * j], pd[4 * j + 1],
                 pd[4 * j + 2], pd[4 * j + 3]);
      };
      auto run_half = [&](auto masked) {
        run_part(0, masked);
        run_part(1, masked);
      };

      if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_ST_DONE + x), it & 1, s_abort))) { ok = false; break; }
      tc_fence_after();
      if (need_mask) run_half(std::true_type{}); else run_half(std::false_type{});
      // On behalf of the MMA warp (see there): this half of the next tile's Q / dO has landed and, half b, the dQ buffer is
      // free.  Neither barrier can be more than one completion ahead: the next fill of that stage and the next dQ both
      // need this arrival first.  (The dS buffer was free: S^T of this tile is complete, hence the dQ MMAs issued before it,
      // those of tile it - 2 among them.)
      bool w2 = it + 1 >= n_iter || mbar_wait_bounded(bar(BAR_Q_FULL + 2 * ((it + 1) & 1) + x), ((it + 1) >> 1) & 1, s_abort);
      if (x == 1 && it > 0 && w2) w2 = mbar_wait_bounded(bar(BAR_DQ_FREE), (it - 1) & 1, s_abort);
      if (!__all_sync(0xffffffffu, w2)) { ok = false; break; }
      fence_proxy_async();          // the dS tile was written with ordinary stores and is read by the MMA
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(BAR_PD_READY + x));
      if (++r_it == nm) { r_it = 0; ++hq_it; }
    }

    // every MMA of the item is complete (a barrier of its own: half a's warps can be two completions ahead of DQ_DONE)
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar(BAR_ACC_DONE), 0, s_abort));
    // dK, dV: rows = keys, all 64 columns of one of them per warp.  The tiles go through shared memory (the Q stages, which
    // nothing reads any more) so that each store instruction writes four whole 128-byte rows: straight from the TMEM
    // layout a warp would touch 32 different rows per instruction, which took 3600 clk per CTA.
    if (ok) {
      tc_fence_after();
      // half a's warps have dK, half b's dV
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + (x == 0 ? cDK : cDV) + hf * 32, r);
        tc_wait_ld();
        if constexpr (PARTS) {
          // fp32, straight from the registers: a row each, 128 bytes of it at a time
          if (n0 + rloc < S) {
            float4* pt = reinterpret_cast<float4*>(part_row(x, n0 + rloc) + hf * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              pt[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
          }
        } else {
          const uint32_t srow = smem_u32(sQ) + x * kTileBytes + rloc * 128;
          const float f = x == 0 ? p.scale : 1.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int i = 8 * j;
            sts_v4(srow + static_cast<uint32_t>(((hf * 4 + j) ^ (rloc & 7)) << 4), pack16b<DT>(__uint_as_float(r[i]) * f, __uint_as_float(r[i + 1]) * f),
                   pack16b<DT>(__uint_as_float(r[i + 2]) * f, __uint_as_float(r[i + 3]) * f),
                   pack16b<DT>(__uint_as_float(r[i + 4]) * f, __uint_as_float(r[i + 5]) * f),
                   pack16b<DT>(__uint_as_float(r[i + 6]) * f, __uint_as_float(r[i + 7]) * f));
          }
        }
      }
    }
    // all eight compute warps pass here, whatever happened before (a named barrier has no time-out)
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
    if (!PARTS && ok) {
      // warp w writes rows 16w .. 16w+15 of both tiles: lane = (row & 3, 16-byte chunk)
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int r = warp * 16 + r4 * 4 + (lane >> 3), c = lane & 7;
        const uint32_t sa = smem_u32(sQ) + r * 128 + static_cast<uint32_t>((c ^ (r & 7)) << 4);
        uint4 vk, vv;
        lds_v4u(sa, vk.x, vk.y, vk.z, vk.w);
        lds_v4u(sa + kTileBytes, vv.x, vv.y, vv.z, vv.w);
        if (n0 + r < S) {
          const int64_t o = bb * p.dk_bs + kvh * p.dk_hs + static_cast<int64_t>(k_begin + n0 + r) * p.dk_rs + c * 8;
          *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.dk) + o) = vk;
          *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.dv) + o) = vv;
        }
      }
    }
    }  // n_iter > 0
  }

  // ---- end of the item: every MMA has completed (the compute warps saw ACC_DONE), every copy has left
  // shared memory; the barriers may be set up again
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  }  // work items

  // ---- teardown ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (tid == 0 && *s_abort != 0) atomicOr(&g_kernel_status, 1);
}

bool make_map64(CUtensorMap* m, int dtype, const void* base, int rows, int H, int B, int64_t rs, int64_t hs, int64_t bs, uint32_t box_rows) {
  const uint64_t dims[4] = {static_cast<uint64_t>(HD), static_cast<uint64_t>(rows), static_cast<uint64_t>(H),
                            static_cast<uint64_t>(B)};
  const uint64_t strides[3] = {static_cast<uint64_t>(rs) * 2, static_cast<uint64_t>(hs) * 2, static_cast<uint64_t>(bs) * 2};
  const uint32_t box[4] = {64, box_rows, 1, 1};
  return encode_tmap(m, dtype == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims,
                     strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

bool bwd_sm100_supported(int dtype, int D) { return (dtype == 0 || dtype == 1) && D == HD && get_encode_tiled() != nullptr; }

// What the tcgen05 backward kernels take beyond dtype and head_dim.  TMA strides must be positive: broadcast
// (stride 0) batch / head dimensions of extent > 1 take the portable kernel.  ALiBi / block mask: dense layout, without
// soft cap or window, mask cells of 32k queries x 16 / 32 / 64 keys.
bool bwd_sm100_strides_ok(const BwdParams& p) {
  if (p.alibi != nullptr || p.bmask != nullptr) {
    if (p.softcap > 0.f || p.window_left >= 0 || p.cu_q != nullptr) return false;
    if (p.bmask != nullptr && (p.bm_bq <= 0 || p.bm_bq % 32 != 0 || !(p.bm_bk == 16 || p.bm_bk == 32 || p.bm_bk == 64))) return false;
  }
  return !((p.B > 1 && (p.q_bs == 0 || p.k_bs == 0 || p.v_bs == 0)) || (p.Hq > 1 && p.q_hs == 0) ||
           (p.Hkv > 1 && (p.k_hs == 0 || p.v_hs == 0)));
}

// The kernel of this file also divides L by the scale (see l_part), which has to leave it a float, and in float16 a number of
// at most 2^31 (Parts3).  What is not an ordinary scale takes the portable kernel.  In float16 that is one below 2^-7 in the log2
// domain: from there on a score of 2^31 times the scale is 2^24 or more, where float32 rounds it by up to 1 and P is off by a
// factor of two in any kernel; below, such scores (rows of a few thousand under a small scale) still have exact gradients.
bool bwd_sm100_takes(const BwdParams& p, int dtype, int D) {
  const float c = fabsf(p.scale_log2);
  return bwd_sm100_supported(dtype, D) && bwd_sm100_strides_ok(p) && (p.softcap > 0.f || (c >= (dtype == 0 ? 0x1p-7f : 1e-6f) && c <= 1e6f));
}

// Main backward step only: p.delta and p.dq_acc must already hold delta and zeros.
cudaError_t launch_bwd_sm100_main(const BwdParams& p, int dtype, int nbatch, int max_k, cudaStream_t stream) {
  if (nbatch <= 0 || max_k <= 0) return cudaSuccess;
  CUtensorMap tmQ, tmK, tmV, tmDO;
  auto fix = [](int64_t s, int64_t fallback) { return s > 0 ? s : fallback; };
  const int64_t q_hs = fix(p.q_hs, static_cast<int64_t>(p.N) * p.q_rs), q_bs = fix(p.q_bs, q_hs * p.Hq);
  const int64_t k_hs = fix(p.k_hs, static_cast<int64_t>(p.S) * p.k_rs), k_bs = fix(p.k_bs, k_hs * p.Hkv);
  const int64_t v_hs = fix(p.v_hs, static_cast<int64_t>(p.S) * p.v_rs), v_bs = fix(p.v_bs, v_hs * p.Hkv);
  const int64_t do_hs = static_cast<int64_t>(p.N) * HD, do_bs = do_hs * p.Hq;
  if (!make_map64(&tmQ, dtype, p.q, p.N, p.Hq, p.B, p.q_rs, q_hs, q_bs, 64) ||
      !make_map64(&tmK, dtype, p.k, p.S, p.Hkv, p.B, p.k_rs, k_hs, k_bs, 128) ||
      !make_map64(&tmV, dtype, p.v, p.S, p.Hkv, p.B, p.v_rs, v_hs, v_bs, 128) ||
      !make_map64(&tmDO, dtype, p.dout, p.N, p.Hq, p.B, HD, do_hs, do_bs, 64))
    return cudaErrorInvalidValue;
  // fp32 dQ accumulator [B][Hq][N][64]: boxes of 32 rows x 32 columns (128 bytes), 128B-swizzled in shared memory
  CUtensorMap tmDQ;
  {
    const uint64_t dims[4] = {static_cast<uint64_t>(HD), static_cast<uint64_t>(p.N), static_cast<uint64_t>(p.Hq),
                              static_cast<uint64_t>(p.B)};
    const uint64_t strides[3] = {static_cast<uint64_t>(HD) * 4, static_cast<uint64_t>(p.N) * HD * 4,
                                 static_cast<uint64_t>(p.Hq) * p.N * HD * 4};
    const uint32_t box[4] = {32, 32, 1, 1};
    if (!encode_tmap(&tmDQ, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p.dq_acc, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return cudaErrorInvalidValue;
  }
  BwdArgs a;
  a.p = p;
  a.dtype = dtype;
  a.gx = (max_k + BK - 1) / BK;
  a.gy = p.Hkv;
  a.parts = p.dkv_part != nullptr ? bwd_dkv_parts(p, p.cu_k != nullptr) : 1;
  a.part = p.dkv_part;
  const long long items = static_cast<long long>(a.gx) * a.gy * nbatch * a.parts;
  if (items > 0x7fffffffLL || p.work_counter == nullptr) return cudaErrorInvalidValue;
  a.total_items = static_cast<int>(items);
  // an item streams Q and dO of one query head at a time
  a.group = p.cu_q != nullptr ? kPackedGroup : order_group(p.causal != 0, p.window_left, static_cast<long long>(p.N) * HD * 4, items / a.gx);
  a.counter = p.work_counter;
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count <= 0) sm_count = 148;
  }
  dim3 grid(static_cast<unsigned>(items < sm_count ? items : sm_count), 1, 1);   // one persistent CTA per SM
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    kern<<<grid, kThreads, kSmemBytes, stream>>>(tmQ, tmK, tmV, tmDO, tmDQ, a);
    return cudaGetLastError();
  };
  const bool cap = p.softcap > 0.f, win = p.window_left >= 0, feat = p.alibi != nullptr || p.bmask != nullptr;
  auto pick = [&](auto parts) -> cudaError_t {
    constexpr bool P = decltype(parts)::value;
    if (feat) return dtype == 0 ? launch(bwd_sm100_kernel<0, false, false, true, P>) : launch(bwd_sm100_kernel<1, false, false, true, P>);
    if (dtype == 0) {
      if (cap) return win ? launch(bwd_sm100_kernel<0, true, true, false, P>) : launch(bwd_sm100_kernel<0, true, false, false, P>);
      return win ? launch(bwd_sm100_kernel<0, false, true, false, P>) : launch(bwd_sm100_kernel<0, false, false, false, P>);
    }
    if (cap) return win ? launch(bwd_sm100_kernel<1, true, true, false, P>) : launch(bwd_sm100_kernel<1, true, false, false, P>);
    return win ? launch(bwd_sm100_kernel<1, false, true, false, P>) : launch(bwd_sm100_kernel<1, false, false, false, P>);
  };
  return a.parts > 1 ? pick(std::true_type{}) : pick(std::false_type{});
}

cudaError_t bwd_sm100_read_clear_status(cudaStream_t stream, int* out) {
  const int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbolAsync(out, g_kernel_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess && *out != 0)
    e = cudaMemcpyToSymbolAsync(g_kernel_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  return e;
}

}  // namespace b200fa
