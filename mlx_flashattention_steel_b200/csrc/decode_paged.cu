// Paged-KV decode: split-KV flash-decoding, its partials merged by their log-sum-exp in
// a dependent kernel.  Replaces the reference's gather + per-sequence two-kernel flash-decode
// route (mlx_mfa/attention.py:3008-3017; csrc/mfa_attention.cpp:150-288; kernels
// csrc/mfa_steel_fwd.cpp:1541-1991, 2008-2105) and its paged forward
// (csrc/mfa_steel_fwd.cpp:2462-3121).
//
// Shape of the work
//   * The pages of all sequences form one list of U units.  CTA c of G takes units
//     [c*U/G, (c+1)*U/G): equal bytes per CTA whatever the sequence lengths are.
//   * A CTA holds HPC kv heads (one consumer warp each) plus one producer warp.  The
//     producer looks pages up in block_table and brings each page in with ONE TMA
//     tensor copy per pool ([block_size tokens] x [HPC heads] x [row bytes], a
//     contiguous 16 KB of HBM for 8 int8 heads), 128B-swizzled by token, plus one
//     bulk copy per scale array, into a ring of stages guarded by mbarriers.
//   * A consumer warp computes S = Q.K^T (rows = the GQA group x query tokens, padded
//     to the 16 rows of mma.m16n8k16) and O^T += V^T.P^T for its head.  8-bit values
//     are widened to f16 in registers straight from the swizzled tile, except for int8
//     K, which meets fixed-point queries on the integer tensor cores; k_scale
//     multiplies the scores, v_scale is folded into P.
//   * A CTA that covers a whole sequence writes the result; otherwise it writes a
//     partial (normalised O, base-2 lse), and a second kernel merges the partials of
//     every row.  Both are launched as programmatic dependents: their blocks take their places while the kernel in
//     front drains (back-to-back calls of 512 int8 tokens 14.5 -> 12.2 us, 262144 tokens 100.9 -> 97.6).  Nobody spins on
//     anybody.
//
//   * Pages of 32, 64, ... tokens are walked as 16-token units (a unit is what one TMA box and one consumer step
//     cover).  Dense caches [B, Hkv, S, D] (the reference's flash-decode route for N <= 4, S >= 256 on plain
//     flash_attention calls, csrc/mfa_attention.cpp:150-288) run the same kernel: unit j of sequence b is its tokens
//     [16 j, 16 j + 16), addressed through a tensor map with the cache's own strides, and no table is read.
//   * head_dim 128 for every pool type; head_dim 64 for 16-bit pools and dense caches.
//
// Every mbarrier wait is bounded (tma.cuh); a timeout raises the error word at the
// start of the workspace (through the merge kernel) and the CTA leaves.
#include <cuda_fp8.h>

#include <cstdio>
#include <type_traits>

#include <mutex>

#include "../../include/b200fa.h"
#include "common.cuh"
#include "decode.h"
#include "tma.cuh"

namespace b200fa {

namespace {

constexpr int kBS = 16;           // tokens per unit (one TMA box, one consumer step); a page is 1, 2, 4, ... units
constexpr int kMaxStages = 8;
constexpr int kMaxWarps = 17;     // warps of a CTA: up to 16 consumers and the producer
// Up to this many sequences every CTA makes the page prefix sums itself, in shared memory (at most 4 KB): one read of
// seq_lens and a scan, ~1 us, where a planning kernel in front and a binary search through its result in global memory
// cost ~6 us before the first page was requested.  Beyond it decode_plan_kernel scans once for all.
constexpr int kSmemSeqs = 1024;
// CTAs that share an SM when a CTA holds few heads: as many as make 8 consumer warps (6 CTAs of one, whose registers
// would otherwise not fit).  The grid counts on all of them being resident at once, hence the launch bounds and the room
// that launch_decode_paged leaves in shared memory.
__host__ __device__ constexpr int ctas_per_sm(int warps) { return warps >= 8 ? 1 : (warps >= 4 ? 2 : (warps >= 2 ? 4 : 6)); }

enum KvKind { KV_F16 = 0, KV_BF16 = 1, KV_I8 = 2, KV_E4M3 = 3 };

struct DecodeLayout {          // workspace carve-up, in bytes from the workspace base
  size_t err;                  // int[4]: [0] error word
  size_t status;               // int[gx * HG * warps of a CTA]: error bits of every warp of the main kernel
  size_t page_start;           // int[B + 1], only when B > kSmemSeqs
  size_t part_lse;             // float[slots * Hq * Nq]
  size_t part_o;               // float[slots * Hq * Nq * D]
  size_t total;
  int slots;
};

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

__host__ __device__ inline DecodeLayout make_layout(int B, int Hq, int Nq, int HG, int G, int kD, int PG) {
  DecodeLayout L;
  L.err = 0;
  L.status = 16;
  L.slots = (G + B) * PG;
  L.page_start = align_up(L.status + sizeof(int) * static_cast<size_t>(G) * HG * kMaxWarps, 16);
  L.part_lse = align_up(L.page_start + (B > kSmemSeqs ? sizeof(int) * (static_cast<size_t>(B) + 1) : 0), 16);
  L.part_o = align_up(L.part_lse + sizeof(float) * static_cast<size_t>(L.slots) * Hq * Nq, 16);
  L.total = align_up(L.part_o + sizeof(float) * static_cast<size_t>(L.slots) * Hq * Nq * kD, 16);
  return L;
}

struct KernelArgs {
  DecodeParams p;
  DecodeLayout lay;
  int HG;            // head groups = Hkv / HPC
  int group;         // Hq / Hkv
  int rows;          // group * Nq
  int hpc;           // kv heads per CTA
  int aligned;       // CTAs of one sequence each (take_aligned)
  int row_groups;    // consumer warps per kv head that share its rows (1 up to 16 rows)
  int page_groups;   // consumer warps per kv head that take its units in turn, each leaving partials of its own
  int stages;
  int upp;              // 16-token units per page = block_size / 16
  int stage_kv_bytes;   // bytes of one K (or V) stage tile = HPC * kBS * row_bytes
  int scale_bytes;      // bytes of one scale page = kBS * Hkv * 2 (0 when not quantized)
  int qlo_bytes;        // int8 pools: low bytes of Q, 1 KB per consumer warp and row tile
  float q_prescale;     // folded into Q (8-bit pools) or applied to the scores (16-bit pools)
  float cap_log2;       // softcap * log2(e)
  float inv_cap;        // 1 / softcap
};

// ---------------------------------------------------------------------------
// plan: page prefix sums of more than kSmemSeqs sequences
// ---------------------------------------------------------------------------
__device__ __forceinline__ int units_of(const int32_t* seq_lens, int i, int max_kv_len) {
  int len = seq_lens != nullptr ? seq_lens[i] : max_kv_len;
  len = len < 0 ? 0 : (len > max_kv_len ? max_kv_len : len);
  return (len + kBS - 1) / kBS;
}

// CTAs (of gx) that work on U units of B sequences.  With few units not every CTA does: two units (one step of the
// consumers) each, or one sequence each when they are that short -- a CTA more to a sequence is a part more to merge, a
// second sequence in a CTA costs it 4 us.  The CTAs that share a sequence are always consecutive.
__host__ __device__ inline int working_ctas(long long U, int B, int gx) {
  const long long pairs = (U + 1) / 2, seqs = U < B ? U : B, want = pairs > seqs ? pairs : seqs;
  return want < static_cast<long long>(gx) ? static_cast<int>(want) : gx;
}

// Few units: every working CTA has units of one sequence alone, a sequence of n units ceil(n / quota) CTAs that share them
// evenly.  Sharing out the whole list evenly gives some CTAs the end of one sequence and the start of the next, and those set
// the time: the second one's queries, table entries and first page come one after the other, 3 to 4 us, about 6 units'
// worth.  What it costs is up to one CTA per sequence that is not full, U / (gx - B) units per CTA instead of U / gx: taken while
// that is at most 6 units more if all sequences were as long as the longest (which the host knows: a template parameter,
// since code for both in one kernel cost 1 us in calls of either).  32 sequences of 500 to 1500 int8 tokens 28.5 -> 27.7 us, 2 of 4000 to
// 16000 with 2 kv heads 18.7 -> 16.2, 16 with 4 queries each 30.6 -> 29.6.
constexpr int kAlignedSeqs = 64;      // two to a lane
inline bool take_aligned(int B, int max_kv_len, int gx) {
  const long long U = static_cast<long long>(B) * ((max_kv_len + kBS - 1) / kBS);
  return B >= 2 && B <= kAlignedSeqs && 2 * B <= gx && U * B <= 6LL * gx * (gx - B);
}
__device__ __forceinline__ int aligned_quota(long long U, int B, int gx) {
  const int q = static_cast<int>((U + gx - B - 1) / (gx - B));
  return q < 2 ? 2 : q;                // one step of the consumers is two units
}
// The CTAs of up to kAlignedSeqs sequences, by a whole warp: lane l has sequences l and l + 32
struct AlignedShares {
  int n0, n1;             // CTAs of them
  int x0, x1;             // CTAs up to and including them
};
__device__ __forceinline__ AlignedShares aligned_shares(const int32_t* seq_lens, int B, int max_kv_len, int quota, int lane) {
  AlignedShares s;
  s.n0 = lane < B ? (units_of(seq_lens, lane, max_kv_len) + quota - 1) / quota : 0;
  s.n1 = lane + 32 < B ? (units_of(seq_lens, lane + 32, max_kv_len) + quota - 1) / quota : 0;
  s.x0 = s.n0;
  s.x1 = s.n1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y0 = __shfl_up_sync(0xffffffffu, s.x0, o), y1 = __shfl_up_sync(0xffffffffu, s.x1, o);
    if (lane >= o) { s.x0 += y0; s.x1 += y1; }
  }
  s.x1 += __shfl_sync(0xffffffffu, s.x0, 31);
  return s;
}

__global__ void __launch_bounds__(1024) decode_plan_kernel(const int32_t* __restrict__ seq_lens, int B, int max_kv_len,
                                                           int* __restrict__ page_start) {
  __shared__ int warp_sums[32];
  __shared__ int carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) { carry = 0; page_start[0] = 0; }
  __syncthreads();
  for (int base = 0; base < B; base += blockDim.x) {
    const int i = base + tid;
    int x = i < B ? units_of(seq_lens, i, max_kv_len) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sums[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const int incl = x + (warp > 0 ? warp_sums[warp - 1] : 0) + carry;
    if (i < B) page_start[i + 1] = incl;
    __syncthreads();
    if (tid == blockDim.x - 1) carry = incl;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};\n" ::"r"(addr), "r"(x), "r"(y));
}
__device__ __forceinline__ float lds_half(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(addr));
  return __half2float(__ushort_as_half(v));
}
// two biased bytes (x ^ 0x80) at byte positions given by `sel` -> half2 of the signed values
__device__ __forceinline__ uint32_t i8pair_to_h2(uint32_t biased, uint32_t sel) {
  const uint32_t magic = prmt(biased, 0x64646464u, sel);      // 0x64XX64YY = 1024 + u
  __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&magic), __floats2half2_rn(1152.f, 1152.f));
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t e4m3pair_to_h2(uint32_t two_bytes) {
  __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(two_bytes & 0xffffu), __NV_E4M3);
  __half2 h = r;
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// D (16 x 8, int32) += A (16 x 32, int8) B (32 x 8, int8).  8.3 clk per instruction and scheduler, what the f16
// m16n8k16 takes (8.4), for twice the depth.
__device__ __forceinline__ void mma16832_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float clamp_h(float x) { return fabsf(x) <= 3.4028235e38f ? fminf(fmaxf(x, -65504.f), 65504.f) : NAN; }

// CTA index (of G) whose unit range [c*U/G, (c+1)*U/G) holds unit u
__device__ __forceinline__ int cta_of_unit(long long u, int G, long long U) {
  return static_cast<int>(((u + 1) * G - 1) / U);
}

// ---------------------------------------------------------------------------
// merge of partials
// ---------------------------------------------------------------------------
// L = log2 sum_i 2^lse_i, O = sum_i 2^(lse_i - L) O_i over the parts of a sequence (csrc/mfa_steel_fwd.cpp:2066-2101);
// rows of empty sequences become zeros with lse = -inf.  A block of max(8, W) warps holds rows of which W warps each take the
// parts in turn; lane l carries head-dim values [4l, 4l + 4).  Bound by L2 latency: a warp asks for its log-sum-exps
// and for its first partial rows at the same time, and W is such that a sequence of average length has few more
// parts per warp.  (With the log-sum-exps first, 6 rows at a time and at most 8 warps, one sequence of 262144 tokens
// in 296 parts was merged 10 us after the main kernel's end, now 5.5; a call 105.8 -> 100.9 us, 8 sequences of 100 to 1000
// tokens 20.6 -> 18.6.)  The first version
// merged inside the main kernel, in the CTA that arrived last (fences, an atomic, then one SM's eight warps for every row):
// 262144 tokens in 148 parts 198 us in all, 512 tokens 21 us of which 13 were the merge.  Here every row has warps of its
// own, and the block knows its sequence's parts when the main kernel ends.
constexpr int kMergeWarps = 8;         // warps of a block, unless a row has more
constexpr int kMaxMergeWarps = 32;

// AL: the main kernel's CTAs have one sequence each.  MANY: W > 1.  One warp to a row has few parts: 6 at a time, and four blocks to an SM.
template <int kD, bool MANY, bool AL>
__global__ void __launch_bounds__(MANY ? kMaxMergeWarps * 32 : kMergeWarps * 32, MANY ? 1 : 4)
decode_merge_kernel(const __grid_constant__ KernelArgs a, int gx, int W_, int blocks_per_seq, int let_in) {
  constexpr int kBatch = MANY ? 8 : 6;                // partial rows in flight per warp
  const int W = MANY ? W_ : 1;
  const DecodeParams& p = a.p;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x / blocks_per_seq;
  unsigned char* ws = reinterpret_cast<unsigned char*>(p.workspace);
  __shared__ int s_sum[2][kMaxMergeWarps];
  __shared__ float2 s_part[kMaxMergeWarps];
  extern __shared__ float4 s_acc[];                   // [warps][32], W > 1
  const int warps = MANY ? static_cast<int>(blockDim.x) >> 5 : kMergeWarps;

  // units before sequence b, and of all: up to kSmemSeqs sequences from the lengths, which are inputs of the launch, so
  // that there is nothing to wait for; beyond from the plan kernel's sums (a scan per block would be quadratic in B)
  long long s0 = 0, U = 0;
  if (p.B <= kSmemSeqs) {
    int before = 0, all = 0;
    for (int i = tid; i < p.B; i += blockDim.x) {
      const int n = units_of(p.seq_lens, i, p.max_kv_len);
      all += n;
      if (i < b) before += n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (lane == 0) { s_sum[0][warp] = before; s_sum[1][warp] = all; }
    __syncthreads();
    for (int i = 0; i < warps; ++i) { s0 += s_sum[0][i]; U += s_sum[1][i]; }
  } else {
    pdl_wait();
    const int* page_start = reinterpret_cast<const int*>(ws + a.lay.page_start);
    s0 = __ldcg(page_start + b);
    U = __ldcg(page_start + p.B);
  }
  const int n_units = units_of(p.seq_lens, b, p.max_kv_len);
  int c_first = 0, n = 0;
  if constexpr (AL) {
    const AlignedShares s = aligned_shares(p.seq_lens, p.B, p.max_kv_len, aligned_quota(U, p.B, gx), lane);
    n = __shfl_sync(0xffffffffu, b < 32 ? s.n0 : s.n1, b & 31);
    c_first = __shfl_sync(0xffffffffu, b < 32 ? s.x0 : s.x1, b & 31) - n;
  } else if (n_units > 0) {
    const int G = working_ctas(U, p.B, gx);
    c_first = cta_of_unit(s0, G, U);
    n = cta_of_unit(s0 + n_units - 1, G, U) - c_first + 1;
  }

  pdl_wait();               // the main kernel has ended: its partials and status words can be read
  if (let_in) pdl_launch_dependents();

  if (blockIdx.x == 0) {
    // error word = all bits that the main kernel's warps left
    const int* status = reinterpret_cast<const int*>(ws + a.lay.status);
    const int words = gx * a.HG * (a.hpc * a.row_groups * a.page_groups + 1);
    int bits = 0;
    for (int i = tid; i < words; i += blockDim.x) bits |= __ldcg(status + i);
    bits = __reduce_or_sync(0xffffffffu, bits);
    __syncthreads();
    if (lane == 0) s_sum[0][warp] = bits;
    __syncthreads();
    if (tid == 0) {
      for (int i = 1; i < warps; ++i) bits |= s_sum[0][i];
      *reinterpret_cast<int*>(ws + a.lay.err) = bits;
    }
  }
  if (a.page_groups == 1 && n == 1) return;           // one CTA had the whole sequence and wrote the result
  n *= a.page_groups;

  const int HqNq = p.Hq * p.Nq;
  const int sub = warp % W;                           // which of the row's warps
  const int row = (blockIdx.x % blocks_per_seq) * (warps / W) + warp / W;            // hq * Nq + query token
  const bool live = lane * 4 < kD;                    // head_dim 64: the first 16 lanes carry the row
  float m = -INFINITY, wsum = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row < HqNq) {
    const size_t slot0 = (static_cast<size_t>(c_first) + b) * a.page_groups;
    const float* lse = reinterpret_cast<const float*>(ws + a.lay.part_lse) + slot0 * HqNq + row;
    const float* o = reinterpret_cast<const float*>(ws + a.lay.part_o) + (slot0 * HqNq + row) * kD + lane * 4;
    const size_t o_step = static_cast<size_t>(HqNq) * kD;
    // this warp's parts: sub, sub + W, ...; 32 of them at a time
    for (int base = sub; base < n; base += 32 * W) {
      const int cn = min(32, (n - base + W - 1) / W);
      float4 v[kBatch];
      auto fetch = [&](int i0) {
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (live && i0 + k < cn) v[k] = __ldcg(reinterpret_cast<const float4*>(o + static_cast<size_t>(base + (i0 + k) * W) * o_step));
        }
      };
      const float lv = lane < cn ? __ldcg(lse + static_cast<size_t>(base + lane * W) * HqNq) : -INFINITY;
      fetch(0);
      float mx = lv;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
      const float m_new = fmaxf(m, mx);
      const float ms = (m_new == -INFINITY) ? 0.f : m_new;
      const float corr = exp2f(m - ms);               // 0 from -inf
      acc.x *= corr; acc.y *= corr; acc.z *= corr; acc.w *= corr;
      const float w = exp2f(lv - ms);
      float sum = w;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
      wsum = fmaf(wsum, corr, sum);
      m = m_new;
      for (int i0 = 0; i0 < cn; i0 += kBatch) {
        if (i0 > 0) fetch(i0);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const float wk = __shfl_sync(0xffffffffu, w, (i0 + k) & 31);
          acc.x = fmaf(wk, v[k].x, acc.x); acc.y = fmaf(wk, v[k].y, acc.y);
          acc.z = fmaf(wk, v[k].z, acc.z); acc.w = fmaf(wk, v[k].w, acc.w);
        }
      }
    }
  }
  if constexpr (MANY) {
    s_acc[warp * 32 + lane] = acc;
    if (lane == 0) s_part[warp] = make_float2(m, wsum);
    __syncthreads();
    if (sub != 0) return;
    // lane i: what the row's warp i has; one pass over their accumulators
    const float2 pi = lane < W ? s_part[warp + lane] : make_float2(-INFINITY, 0.f);
    m = pi.x;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    const float wi = exp2f(pi.x - (m == -INFINITY ? 0.f : m));
    wsum = wi * pi.y;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, s);
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int i = 0; i < W; ++i) {
      const float c = __shfl_sync(0xffffffffu, wi, i);
      const float4 v = s_acc[(warp + i) * 32 + lane];
      acc.x = fmaf(c, v.x, acc.x); acc.y = fmaf(c, v.y, acc.y); acc.z = fmaf(c, v.z, acc.z); acc.w = fmaf(c, v.w, acc.w);
    }
  }
  if (row >= HqNq) return;
  const float inv = wsum > 0.f ? 1.f / wsum : 0.f;
  const float lse = wsum > 0.f ? m + log2f(wsum) : -INFINITY;
  const float4 v = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
  const size_t orow = static_cast<size_t>(b) * HqNq + row;
  if (p.packed_f32) {
    float* pk = reinterpret_cast<float*>(p.out) + orow * (kD + 4);
    if (live) *reinterpret_cast<float4*>(pk + lane * 4) = v;
    if (lane == 0) pk[kD] = lse;
  } else {
    if (live) {
      const uint2 pk = p.q_dtype == 0 ? make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w)) : make_uint2(pack_bf2(v.x, v.y), pack_bf2(v.z, v.w));
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.out) + orow * kD + lane * 4) = pk;
    }
    if (p.lse != nullptr && lane == 0) p.lse[orow] = lse;
  }
}

// ---------------------------------------------------------------------------
// main kernel
// ---------------------------------------------------------------------------
// CAP: soft cap on.  A template parameter so that the common launch without one carries no tanh code in its unrolled
// inner loops (with it compiled in, config 4 -- which has no soft cap -- ran 4 % slower).
// RT: tiles of 8 query rows (of the group's heads x query tokens) per consumer warp.  RT = 1: up to 8 rows, one warp per
// kv head, HPC heads per CTA.  RT = 2 (HPC = 0: a.hpc heads, known at run time): up to 16 rows per warp, which fills the
// 16 rows of the MMA, and a.row_groups warps per head share a page when there are more.
// PG = 2: two warps per head take its units in turn (one each step instead of two), which doubles the warps that hide the
// latency of a step's chain of waits, conversions and MMAs.
// Launch bounds: those of the CTA's own width, or for RT = 2, whose width is known at run time, 384 threads (168
// registers a thread: 2 CTAs of 5 warps, 4 of 3 or 6 of 2 fit an SM's 65536).
template <int KV, int HPC, int kD, bool CAP, int RT, int PG, bool AL>
__global__ void __launch_bounds__(HPC > 0 ? (HPC * PG + 1) * 32 : 384, HPC > 0 ? ctas_per_sm(HPC) : 1)
decode_paged_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const KernelArgs a) {
  constexpr bool kQuant = (KV == KV_I8 || KV == KV_E4M3);
  static_assert(kD == 128 || (kD == 64 && !kQuant), "head_dim 64 is built for 16-bit pools only");
  constexpr int kKS = kD / 16;                         // k-steps of S = Q.K^T, m-tiles of O^T
  constexpr int kRowBytes = kQuant ? kD : 2 * kD;      // bytes of one (token, head) row
  constexpr int kHeadBytes = kBS * kRowBytes;          // one head of one page in shared memory
  using MmaT = typename std::conditional<KV == KV_BF16, __nv_bfloat16, __half>::type;

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // carve: [stages] K tiles, [stages] V tiles, [stages] k scales, [stages] v scales, low bytes of Q, barriers, misc
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const DecodeParams& p = a.p;
  const int NS = a.stages;
  unsigned char* sK = smem;
  unsigned char* sV = sK + static_cast<size_t>(NS) * a.stage_kv_bytes;
  unsigned char* sKs = sV + static_cast<size_t>(NS) * a.stage_kv_bytes;
  unsigned char* sVs = sKs + static_cast<size_t>(NS) * a.scale_bytes;
  unsigned char* s_qlo = sVs + static_cast<size_t>(NS) * a.scale_bytes;      // int8: lo bytes of Q, 1 KB per consumer warp and row tile
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_qlo + a.qlo_bytes);         // full[NS], empty[NS]
  int* s_page = reinterpret_cast<int*>(bars + 2 * kMaxStages);
  volatile int* s_abort = s_page + kMaxStages;
  int* s_page_start = const_cast<int*>(s_abort) + 1;     // int[B + 1] when B <= kSmemSeqs

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int hg = blockIdx.y;
  const int c = blockIdx.x;
  const int hpc = HPC > 0 ? HPC : a.hpc;
  const int n_cons = HPC > 0 ? HPC * PG : a.hpc * a.row_groups;       // consumer warps; the next one is the producer

  unsigned char* ws = reinterpret_cast<unsigned char*>(p.workspace);
  // every warp leaves its error bits (1: a bounded wait gave up, 2: a table entry beyond the pool)
  int* status = reinterpret_cast<int*>(ws + a.lay.status) + (static_cast<size_t>(hg) * gridDim.x + c) * (n_cons + 1) + warp;
  float* part_lse = reinterpret_cast<float*>(ws + a.lay.part_lse);
  float* part_o = reinterpret_cast<float*>(ws + a.lay.part_o);

  const int rows = a.rows;
  const int HqNq = p.Hq * p.Nq;

  if (tid == 0) {
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    for (int i = 0; i < NS; ++i) {
      mbar_init(smem_u32(&bars[i]), 1);                 // full: producer arrive (+ tx bytes)
      mbar_init(smem_u32(&bars[kMaxStages + i]), n_cons / PG);  // empty: one arrive per warp that reads the stage
    }
    *s_abort = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  // The kernel before this one has ended: its outputs (lengths, tables, queries, the rows just appended) can be read.  Only now
  // may the merge kernel's blocks take their places, since they read the lengths without a wait of their own.
  pdl_wait();
  pdl_launch_dependents();
  // page prefix sums
  const int* page_start = s_page_start;
  if (p.B <= kSmemSeqs) {
    for (int i = tid; i < p.B; i += blockDim.x) s_page_start[i + 1] = units_of(p.seq_lens, i, p.max_kv_len);
    __syncthreads();
    if (warp == 0) {
      // lane l owns the entries [l * per, (l + 1) * per)
      const int per = (p.B + 31) >> 5, i0 = lane * per, i1 = min(p.B, i0 + per);
      int sum = 0;
      for (int i = i0; i < i1; ++i) sum += s_page_start[i + 1];
      int x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      x -= sum;
      for (int i = i0; i < i1; ++i) { x += s_page_start[i + 1]; s_page_start[i + 1] = x; }
      if (lane == 0) s_page_start[0] = 0;
    }
  } else {
    page_start = reinterpret_cast<const int*>(ws + a.lay.page_start);
  }
  __syncthreads();

  const long long U = page_start[p.B];
  const int G = AL ? 0 : working_ctas(U, p.B, static_cast<int>(gridDim.x));
  long long lo = 0, hi = 0;
  int b_first = 0, aligned_parts = 0;
  if constexpr (AL) {
    const AlignedShares s = aligned_shares(p.seq_lens, p.B, p.max_kv_len, aligned_quota(U, p.B, static_cast<int>(gridDim.x)), lane);
    // this CTA's sequence: as many as have all their CTAs before it (and an empty one has none)
    b_first = __popc(__ballot_sync(0xffffffffu, lane < p.B && s.x0 <= c)) + __popc(__ballot_sync(0xffffffffu, lane + 32 < p.B && s.x1 <= c));
    if (b_first < p.B) {
      aligned_parts = __shfl_sync(0xffffffffu, b_first < 32 ? s.n0 : s.n1, b_first & 31);
      const int k = c - (__shfl_sync(0xffffffffu, b_first < 32 ? s.x0 : s.x1, b_first & 31) - aligned_parts);
      const int s0 = page_start[b_first], n = page_start[b_first + 1] - s0;
      lo = s0 + static_cast<long long>(k) * n / aligned_parts;
      hi = s0 + static_cast<long long>(k + 1) * n / aligned_parts;
    }
  } else if (c < G) {
    lo = static_cast<long long>(c) * U / G;
    hi = static_cast<long long>(c + 1) * U / G;
  }
  if (lo >= hi) {
    if (lane == 0) *status = 0;
    return;
  }

  // first sequence: largest b with page_start[b] <= lo
  if constexpr (!AL) {
    int l = 0, r = p.B;   // invariant: page_start[l] <= lo < page_start[r]  (page_start[B] = U > lo)
    while (r - l > 1) {
      const int m = (l + r) >> 1;
      if (page_start[m] <= lo) l = m; else r = m;
    }
    b_first = l;
  }

  const uint32_t tx_bytes = 2u * a.stage_kv_bytes + 2u * a.scale_bytes;

  if (warp == n_cons) {
    // ======================= producer warp =======================
    int stage = 0;
    uint32_t phase = 0;
    long long u = lo;
    int b = b_first;
    bool ok = true;
    int bad = 0;
    while (u < hi && ok) {
      const int s0 = page_start[b], s1 = page_start[b + 1];
      if (s1 <= u) { ++b; continue; }
      const int j_lo = static_cast<int>(u - s0);
      const int j_hi = static_cast<int>((hi < s1 ? hi : s1) - s0);
      const int32_t* row = p.dense ? nullptr : p.block_table + static_cast<size_t>(b) * p.max_blocks;
      for (int j0 = j_lo; j0 < j_hi && ok; j0 += 32) {
        const int jj = j0 + lane;
        // first token of unit jj in the pool (paged: its page's tokens start at page * block_size) or in the
        // sequence (dense); -1 = no page
        int my_tok = -1;
        if (jj < j_hi) {
          if (p.dense) {
            my_tok = jj * kBS;
          } else {
            const int pg_id = row[jj / a.upp];
            if (pg_id >= p.num_pages) bad = 2;                       // table entry beyond the pool
            else if (pg_id >= 0) my_tok = pg_id * p.block_size + (jj % a.upp) * kBS;
          }
        }
        const int n = min(32, j_hi - j0);
        for (int i = 0; i < n; ++i) {
          const int page = __shfl_sync(0xffffffffu, my_tok, i);       // token offset of the unit, or -1
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bars[kMaxStages + stage]), phase ^ 1u, s_abort))) { ok = false; break; }
          if (lane == 0) {
            s_page[stage] = page;
            const uint32_t full = smem_u32(&bars[stage]);
            if (page >= 0) {
              mbar_arrive_expect_tx(full, tx_bytes);
              const int batch_coord = p.dense ? b : 0;
              tma_load_5d(smem_u32(sK + static_cast<size_t>(stage) * a.stage_kv_bytes), &tmK, full, 0, page, 0, hg * hpc, batch_coord);
              tma_load_5d(smem_u32(sV + static_cast<size_t>(stage) * a.stage_kv_bytes), &tmV, full, 0, page, 0, hg * hpc, batch_coord);
              if (kQuant) {
                const size_t soff = static_cast<size_t>(page / kBS) * a.scale_bytes;
                bulk_load(smem_u32(sKs + static_cast<size_t>(stage) * a.scale_bytes),
                          reinterpret_cast<const unsigned char*>(p.k_scale) + soff, a.scale_bytes, full);
                bulk_load(smem_u32(sVs + static_cast<size_t>(stage) * a.scale_bytes),
                          reinterpret_cast<const unsigned char*>(p.v_scale) + soff, a.scale_bytes, full);
              }
            } else {
              mbar_arrive(full);                  // hole in the table: consumers treat K = V = 0
            }
          }
          __syncwarp();
          if (++stage == NS) { stage = 0; phase ^= 1u; }
        }
      }
      u = s0 + j_hi;
      if (u >= s1) ++b;
    }
    bad = __reduce_or_sync(0xffffffffu, bad | (ok ? 0 : 1));
    if (lane == 0) *status = bad;
    return;
  }

  // ======================= consumer warps =======================
  static_assert(RT == 1 || PG == 1, "wide rows split a head by rows");
  constexpr int NPI = PG == 1 ? 2 : 1;                          // units per step
  const int pgrp = PG == 1 ? 0 : warp % PG;
  const int wh = RT == 1 ? warp / PG : warp / a.row_groups;          // kv head of this warp within the CTA
  const int rbase = RT == 1 ? 0 : (warp % a.row_groups) * (8 * RT);
  const int kvh = hg * hpc + wh;
  // fragment row g of row tile rt is query row rbase + 8 rt + g = (query token, head of the group)
  int row_of[RT], qi_row[RT], hq_row[RT];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) {
    row_of[rt] = rbase + 8 * rt + g;
    qi_row[rt] = row_of[rt] / a.group;
    hq_row[rt] = kvh * a.group + row_of[rt] % a.group;
  }
  int stage = pgrp;             // the ring has at least two stages
  uint32_t phase = 0;
  long long u = lo;
  int b = b_first;
  bool ok = true;

  while (u < hi && ok) {
    const int s0 = page_start[b], s1 = page_start[b + 1];
    if (s1 <= u) { ++b; continue; }
    // this warp's units: all, or those at its parity of the CTA's running count
    const int j_lo = static_cast<int>(u - s0) + (PG == 1 ? 0 : static_cast<int>((u - lo + pgrp) & 1));
    const int j_hi = static_cast<int>((hi < s1 ? hi : s1) - s0);
    int len = p.seq_lens != nullptr ? p.seq_lens[b] : p.max_kv_len;
    len = len < 0 ? 0 : (len > p.max_kv_len ? p.max_kv_len : len);
    const int n_parts = AL ? aligned_parts : cta_of_unit(static_cast<long long>(s1) - 1, G, U) - cta_of_unit(s0, G, U) + 1;

    // ---- Q fragments (A operand) ----
    // 16-bit and e4m3 pools: qa[s][0 | 1] = row tile 0 (k low, k high), [2 | 3] = row tile 1; kKS k-steps.
    // int8 pools: the products run on the integer tensor cores, K as it is stored (no widening, 3 operations per two
    // values).  A row of Q is fixed point below its largest value: 65536 hi + 256 mid + lo, three signed bytes, in steps
    // of max|q| / 8355000.  hi and mid, whose 256 * hi.k + mid.k is exact in 32 bits (|.| <= 128 * 32639 * 128), are one
    // MMA (one row tile: hi in rows 0..7, mid in rows 8..15) or one each (two row tiles), and their step, 256 times that,
    // is as exact as f16 for values down to a 24th of the largest.  They are enough while at most a quarter of a row's
    // channels lie below that (zeros are exact); else K may be small in the few channels in which Q is large, and lo,
    // from shared memory, joins in another MMA.  128 sequences of 512 to 32768 tokens: 626 us without lo in any row, 687
    // with lo in all.
    constexpr bool kI8 = KV == KV_I8;
    constexpr int kQA = kI8 ? 4 * RT : kKS;
    constexpr int kQR = kI8 ? 4 : 2 * RT;
    uint32_t qa[kQA][kQR];
    float qscale[RT];
    bool fine = false;                            // int8: lo is needed in some row of this warp
    const uint32_t qlo = smem_u32(s_qlo + warp * (RT * 1024));
    __syncwarp();
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      const bool row_valid = row_of[rt] < rows;
      const size_t qoff = row_valid ? ((static_cast<size_t>(b) * p.Hq + hq_row[rt]) * p.Nq + qi_row[rt]) * kD : 0;
      qscale[rt] = 1.f;
      if constexpr (kQuant) {
        // lane t owns d in [32t, 32t+32)
        float f[32];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 w = row_valid ? reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.q) + qoff + 32 * t)[i]
                                    : make_uint4(0u, 0u, 0u, 0u);
          const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 v2 = p.q_dtype == 0 ? __half22float2(*reinterpret_cast<const __half2*>(&ww[e]))
                                             : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ww[e]));
            f[i * 8 + e * 2] = v2.x * a.q_prescale;
            f[i * 8 + e * 2 + 1] = v2.y * a.q_prescale;
          }
        }
        // largest magnitude of the row, as bits: infinities and NaNs are above every number.  Such a row's scores are NaN.
        uint32_t mb = 0u;
        if constexpr (kI8 || RT == 2) {
#pragma unroll
          for (int i = 0; i < 32; ++i) mb = max(mb, __float_as_uint(f[i]) & 0x7fffffffu);
          mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
          mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
        }
        const bool finite = mb < 0x7f800000u;
        if constexpr (kI8) {
          const float mx = __uint_as_float(mb);
          // below 2^-100 the reciprocal would leave the float range; such a row scores zero
          const float inv = finite && mx > 7.9e-31f ? 8355000.f / mx : 0.f;
          qscale[rt] = finite ? mx * (256.f / 8355000.f) : NAN;
          int small = 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) small += (f[i] != 0.f && fabsf(f[i]) < mx * (1.f / 24.f)) ? 1 : 0;
          small += __shfl_xor_sync(0xffffffffu, small, 1);
          small += __shfl_xor_sync(0xffffffffu, small, 2);
          const bool low = finite && small > 32;            // rows that do without have lo = 0: no row's bits depend on another's
          fine = __any_sync(0xffffffffu, fine || low);
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            uint32_t hi4[2], mid4[2], lo4[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              hi4[h] = mid4[h] = lo4[h] = 0u;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int qi = __float2int_rn(f[8 * s + 4 * h + e] * inv);
                const int hb = (qi + 0x8080) >> 16, r = qi - (hb << 16), mib = (r + 0x80) >> 8, lb = r - (mib << 8);
                hi4[h] |= (static_cast<uint32_t>(hb) & 0xffu) << (8 * e);
                mid4[h] |= (static_cast<uint32_t>(mib) & 0xffu) << (8 * e);
                lo4[h] |= (static_cast<uint32_t>(lb) & 0xffu) << (8 * e);
              }
            }
            sts64(qlo + rt * 1024 + (s >> 1) * 512 + lane * 16 + (s & 1) * 8, low ? lo4[0] : 0u, low ? lo4[1] : 0u);
            if constexpr (RT == 1) {
              qa[s][0] = hi4[0]; qa[s][1] = mid4[0]; qa[s][2] = hi4[1]; qa[s][3] = mid4[1];
            } else {
              qa[s][rt] = hi4[0]; qa[s][2 + rt] = hi4[1];
              qa[4 + s][rt] = mid4[0]; qa[4 + s][2 + rt] = mid4[1];
            }
          }
        } else {
          // f16.  Up to 8 rows: values beyond its range become its largest.  More rows, whose calls the prefill kernel
          // ran in the query's own type before: the row over a power of two, its largest value in [2^13, 2^14).
          float down = 1.f;
          if constexpr (RT == 2) {
            const uint32_t ex = min(max(mb >> 23, 15u), 253u);
            down = __uint_as_float((267u - ex) << 23);                          // 2^(13 - (ex - 127))
            qscale[rt] = finite ? __uint_as_float((ex - 13u) << 23) : NAN;
          }
          auto h = [&](float x) { return RT == 2 ? x * down : clamp_h(x); };
          // k-step s uses d = 32t + 4s + {0,1 | 2,3}
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            qa[s][2 * rt] = pack_h2(h(f[4 * s]), h(f[4 * s + 1]));
            qa[s][2 * rt + 1] = pack_h2(h(f[4 * s + 2]), h(f[4 * s + 3]));
          }
        }
      } else {
        // natural order: a0 = Q[g][16s + 2t, +1], a2 = Q[g][16s + 8 + 2t, +1]
        const uint32_t* src = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint16_t*>(p.q) + qoff);
#pragma unroll
        for (int s = 0; s < kKS; ++s) {
          qa[s][2 * rt] = row_valid ? src[8 * s + t] : 0u;
          qa[s][2 * rt + 1] = row_valid ? src[8 * s + 4 + t] : 0u;
        }
      }
    }

    __syncwarp();

    float oacc[RT][kKS][4];
#pragma unroll
    for (int rt = 0; rt < RT; ++rt)
#pragma unroll
      for (int i = 0; i < kKS; ++i) { oacc[rt][i][0] = oacc[rt][i][1] = oacc[rt][i][2] = oacc[rt][i][3] = 0.f; }
    float m_run[RT], l_run[RT];
    int causal_lim[RT];                           // last visible token of the row
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      m_run[rt] = -INFINITY;
      l_run[rt] = 0.f;
      causal_lim[rt] = p.causal ? (qi_row[rt] + len - p.Nq) : 0x7fffffff;
    }
    // Tokens before this one are visible to every row and inside the sequence: steps that end before it need no masks.
    const int open_end = p.causal ? min(len, len - p.Nq + 1) : len;
    // Quantised pools: P goes into its 16-bit operand multiplied by v_scale.  Every exponent is shifted by vexp, minus
    // the exponent of the largest v scale of the first step, so that the product stays inside f16's normal range; the
    // row sum carries the same power of two and it cancels.  A scale of vlimit = 2^(15 - vexp) or more moves vexp, and
    // what has been summed with it, down.
    float vexp = 0.f, vlimit = 0.f;

    // Two pages per iteration: their loads, conversions and MMAs are independent, which gives the
    // scheduler twice the instruction-level parallelism, and one online-softmax step covers 32 tokens.
    // FINE: with lo.  The loop exists twice: lo in a branch inside it cost every call 3 to 5 %.
    auto walk = [&](auto fine_c) __attribute__((always_inline)) {
    constexpr bool FINE = decltype(fine_c)::value;
    for (int j = j_lo; j < j_hi; j += 2) {
      const int np = min(NPI, j_hi - j);
      int stg[NPI], pg[NPI];
      {
        int s2 = stage;
        uint32_t ph2 = phase;
        bool okw = true;
#pragma unroll
        for (int q = 0; q < NPI; ++q) {
          stg[q] = s2;
          if (q < np && okw) {
            okw = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bars[s2]), ph2, s_abort));
            if (++s2 == NS) { s2 = 0; ph2 ^= 1u; }
          }
        }
        if (!okw) { ok = false; break; }
      }
      uint32_t kbase[NPI], vbase[NPI];
#pragma unroll
      for (int q = 0; q < NPI; ++q) {
        pg[q] = q < np ? s_page[stg[q]] : -2;       // -1: hole in the table, -2: no second page
        kbase[q] = smem_u32(sK + static_cast<size_t>(stg[q]) * a.stage_kv_bytes) + wh * kHeadBytes;
        vbase[q] = smem_u32(sV + static_cast<size_t>(stg[q]) * a.stage_kv_bytes) + wh * kHeadBytes;
      }
      // warp-uniform: two pages of visible tokens -- everything below that deals with edges is skipped
      const bool full = (pg[0] | pg[NPI - 1]) >= 0 && (j + NPI) * kBS <= open_end;

      // ---- scales: lane l fetches those of token l & 15 of page l >> 4; shuffles hand them round ----
      float ksl = 1.f, vsl = 0.f;
      bool vmove = false;
      if constexpr (kQuant) {
        const int q = NPI == 2 ? lane >> 4 : 0;
        if (full || (q == 0 ? pg[0] : pg[NPI - 1]) >= 0) {
          const uint32_t off = static_cast<uint32_t>(q == 0 ? stg[0] : stg[NPI - 1]) * a.scale_bytes +
                               static_cast<uint32_t>(((lane & 15) * p.Hkv + kvh) * 2);
          ksl = lds_half(smem_u32(sKs) + off);
          vsl = lds_half(smem_u32(sVs) + off);
        }
        // whatever the scale of a slot beyond the sequence holds (it may be a NaN pattern)
        if (!full && (j + q) * kBS + (lane & 15) >= len) vsl = 0.f;
        vmove = fabsf(vsl) > vlimit && fabsf(vsl) < INFINITY;
      }

      // ---- S = Q K^T : per page this lane gets tokens {2t, 2t+1, 8+2t, 9+2t} of its rows ----
      float sc[RT][NPI][4];
      if constexpr (kI8) {
#pragma unroll
        for (int q = 0; q < NPI; ++q)
#pragma unroll
          for (int jn = 0; jn < 2; ++jn) {
            int acc[RT + 1][4];                               // (hi | mid) or hi, mid; then lo
#pragma unroll
            for (int h = 0; h <= RT; ++h) { acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0; }
            if (pg[q] >= 0) {
              const uint32_t rowa = kbase[q] + (8 * jn + g) * 128;           // token 8 jn + g
              const uint4 w0 = lds128(rowa + (((2 * t) ^ g) << 4));
              const uint4 w1 = lds128(rowa + (((2 * t + 1) ^ g) << 4));
              const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
              for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int h = 0; h < RT; ++h)                                  // RT == 2: acc[0] = hi, acc[1] = mid
                  mma16832_s8(acc[h], qa[4 * h + s], words[2 * s], words[2 * s + 1]);
              if constexpr (FINE) {
#pragma unroll
                for (int s = 0; s < 4; s += 2) {
                  const uint4 a0 = lds128(qlo + s * 256 + lane * 16);
                  const uint4 a1 = RT == 2 ? lds128(qlo + 1024 + s * 256 + lane * 16) : make_uint4(0u, 0u, 0u, 0u);
                  const uint32_t x[4] = {a0.x, a1.x, a0.y, a1.y}, y[4] = {a0.z, a1.z, a0.w, a1.w};
                  mma16832_s8(acc[RT], x, words[2 * s], words[2 * s + 1]);
                  mma16832_s8(acc[RT], y, words[2 * s + 2], words[2 * s + 3]);
                }
              }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
              for (int rt = 0; rt < RT; ++rt) {
                float x = __int2float_rn((acc[0][2 * rt + e] << 8) + (RT == 1 ? acc[0][2 + e] : acc[RT - 1][2 * rt + e]));
                if constexpr (FINE) x = fmaf(__int2float_rn(acc[RT][2 * rt + e]), 1.f / 256.f, x);
                sc[rt][q][2 * jn + e] = x * qscale[rt];
              }
            }
          }
      } else {
        float sacc[NPI][2][4];
#pragma unroll
        for (int q = 0; q < NPI; ++q)
#pragma unroll
          for (int i = 0; i < 2; ++i) { sacc[q][i][0] = sacc[q][i][1] = sacc[q][i][2] = sacc[q][i][3] = 0.f; }
#pragma unroll
        for (int q = 0; q < NPI; ++q) {
          if (pg[q] >= 0) {
            if constexpr (kQuant) {
#pragma unroll
              for (int jn = 0; jn < 2; ++jn) {
                const uint32_t rowa = kbase[q] + (8 * jn + g) * 128;
                const uint4 w0 = lds128(rowa + (((2 * t) ^ g) << 4));
                const uint4 w1 = lds128(rowa + (((2 * t + 1) ^ g) << 4));
                const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                  const uint32_t afrag[4] = {qa[s][0], RT == 2 ? qa[s][2 * (RT - 1)] : 0u, qa[s][1], RT == 2 ? qa[s][2 * (RT - 1) + 1] : 0u};
                  mma16816<MmaT>(sacc[q][jn], afrag, e4m3pair_to_h2(words[s]), e4m3pair_to_h2(words[s] >> 16));
                }
              }
            } else {
#pragma unroll
              for (int s = 0; s < kKS; ++s) {
                uint32_t bfr[4];
                const int tok = (lane & 7) + ((lane >> 4) << 3);
                const int dcol = 16 * s + (((lane >> 3) & 1) << 3);
                const uint32_t addr = kbase[q] + (dcol >> 6) * (kBS * 128) + tok * 128 + ((((dcol & 63) >> 3) ^ (tok & 7)) << 4);
                ldmatrix_x4(bfr, addr);
                const uint32_t afrag[4] = {qa[s][0], RT == 2 ? qa[s][2 * (RT - 1)] : 0u, qa[s][1], RT == 2 ? qa[s][2 * (RT - 1) + 1] : 0u};
                mma16816<MmaT>(sacc[q][0], afrag, bfr[0], bfr[1]);
                mma16816<MmaT>(sacc[q][1], afrag, bfr[2], bfr[3]);
              }
            }
          }
        }
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
          for (int q = 0; q < NPI; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float s = sacc[q][e >> 1][2 * rt + (e & 1)];
              sc[rt][q][e] = !kQuant ? s * a.q_prescale : (RT == 2 ? s * qscale[rt] : s);
            }
      }

      // ---- scale / softcap / masks ----
      float vsc[NPI][4];
#pragma unroll
      for (int q = 0; q < NPI; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tok = ((e >> 1) << 3) + 2 * t + (e & 1);
          if constexpr (kQuant) {
            const float ksv = __shfl_sync(0xffffffffu, ksl, 16 * q + tok);
            vsc[q][e] = __shfl_sync(0xffffffffu, vsl, 16 * q + tok);
#pragma unroll
            for (int rt = 0; rt < RT; ++rt) sc[rt][q][e] *= ksv;
          }
          if constexpr (CAP) {
#pragma unroll
            for (int rt = 0; rt < RT; ++rt)
              sc[rt][q][e] = a.cap_log2 * cap_tanh(sc[rt][q][e] * a.inv_cap, a.inv_cap * kPreciseTanhMinCap <= 1.f);
          }
          if (!full) {
            const int tg = (j + q) * kBS + tok;
#pragma unroll
            for (int rt = 0; rt < RT; ++rt)
              if (!(pg[q] != -2 && tg < len && tg <= causal_lim[rt])) sc[rt][q][e] = -INFINITY;
          }
        }

      // ---- online softmax over the (up to) 32 tokens ----
      float m_new[RT], msub[RT];
      bool grew = false;
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        float mx = fmaxf(fmaxf(sc[rt][0][0], sc[rt][0][1]), fmaxf(sc[rt][0][2], sc[rt][0][3]));
        if (NPI == 2) mx = fmaxf(mx, fmaxf(fmaxf(sc[rt][NPI - 1][0], sc[rt][NPI - 1][1]), fmaxf(sc[rt][NPI - 1][2], sc[rt][NPI - 1][3])));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        m_new[rt] = fmaxf(m_run[rt], mx);
        msub[rt] = (m_new[rt] == -INFINITY) ? 0.f : m_new[rt];
        grew = grew || m_new[rt] > m_run[rt];
      }
      if (__any_sync(0xffffffffu, grew || vmove)) {
        float shift = 0.f;
        if (kQuant && __any_sync(0xffffffffu, vmove)) {
          const unsigned top = __reduce_max_sync(0xffffffffu, vmove ? __float_as_uint(fabsf(vsl)) : 0u);
          shift = 127.f - static_cast<float>(top >> 23) - vexp;
          vexp += shift;
          vlimit = exp2f(15.f - vexp);
        }
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
          const float corr = fast_exp2(m_run[rt] - msub[rt] + shift);       // 1 when nothing changed, 0 from -inf
          l_run[rt] *= corr;
          const float c0 = __shfl_sync(0xffffffffu, corr, (2 * t) * 4);
          const float c1 = __shfl_sync(0xffffffffu, corr, (2 * t + 1) * 4);
#pragma unroll
          for (int i = 0; i < kKS; ++i) {
            oacc[rt][i][0] *= c0; oacc[rt][i][1] *= c1; oacc[rt][i][2] *= c0; oacc[rt][i][3] *= c1;
          }
          m_run[rt] = m_new[rt];
        }
      }
      uint32_t pb[RT][NPI][2];
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        const float sub = kQuant ? msub[rt] - vexp : msub[rt];
#pragma unroll
        for (int q = 0; q < NPI; ++q) {
          float pr[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            pr[e] = fast_exp2(sc[rt][q][e] - sub);
            l_run[rt] += pr[e];
            if (kQuant) pr[e] *= vsc[q][e];
          }
          pb[rt][q][0] = KV == KV_BF16 ? pack_bf2(pr[0], pr[1]) : pack_h2(pr[0], pr[1]);
          pb[rt][q][1] = KV == KV_BF16 ? pack_bf2(pr[2], pr[3]) : pack_h2(pr[2], pr[3]);
        }
      }

      // ---- O^T += V^T P^T : rows = 16 head-dim values per m-tile, cols = query rows ----
#pragma unroll
      for (int q = 0; q < NPI; ++q) {
        if (pg[q] >= 0) {
          // Slots of the last page beyond the sequence's end hold whatever the pool's owner left there; their P is
          // zero, but 0 * NaN (or 0 * inf) would still poison the row, so their V values are cleared as they are
          // loaded.  amask[h]: tokens (2t, 2t+1) for h = 0, (2t+8, 2t+9) for h = 1, one 16-bit lane per token.
          const int tail_from = len - (j + q) * kBS;      // first token of this page that is beyond the sequence
          const bool tail = !full && tail_from < kBS;     // warp-uniform
          uint32_t amask[2] = {0xffffffffu, 0xffffffffu};
          if (tail) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              amask[h] = (2 * t + 8 * h < tail_from ? 0x0000ffffu : 0u) | (2 * t + 8 * h + 1 < tail_from ? 0xffff0000u : 0u);
          }
          if constexpr (kQuant) {
            // lane (g,t) reads the 16 head-dim bytes [16g, 16g + 16) of token rows 2t, 2t+1, 2t+8, 2t+9; m-tile i has
            // dims 16g + 2i (fragment row g) and 16g + 2i + 1 (row g + 8)
            const uint32_t xa = ((g ^ ((2 * t) & 7)) << 4), xb = ((g ^ ((2 * t + 1) & 7)) << 4);
            const uint32_t rA = vbase[q] + (2 * t) * 128;
            const uint4 A4 = lds128(rA + xa), B4 = lds128(rA + 128 + xb), C4 = lds128(rA + 8 * 128 + xa), D4 = lds128(rA + 9 * 128 + xb);
            const uint32_t Aw[4] = {A4.x, A4.y, A4.z, A4.w}, Bw[4] = {B4.x, B4.y, B4.z, B4.w};
            const uint32_t Cw[4] = {C4.x, C4.y, C4.z, C4.w}, Dw[4] = {D4.x, D4.y, D4.z, D4.w};
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              const uint32_t bias = kI8 ? 0x80808080u : 0u;
              const uint32_t A = Aw[jj] ^ bias, B = Bw[jj] ^ bias, Cc = Cw[jj] ^ bias, D = Dw[jj] ^ bias;
              const uint32_t ab[2] = {prmt(A, B, 0x5140u), prmt(A, B, 0x7362u)};   // [A0 B0 A1 B1], [A2 B2 A3 B3]
              const uint32_t cd[2] = {prmt(Cc, D, 0x5140u), prmt(Cc, D, 0x7362u)};
#pragma unroll
              for (int kp = 0; kp < 2; ++kp) {
                uint32_t af[4];
                if (kI8) {
                  af[0] = i8pair_to_h2(ab[kp], 0x4140u);   // head-dim byte 2kp   , tokens 2t, 2t+1
                  af[1] = i8pair_to_h2(ab[kp], 0x4342u);   // head-dim byte 2kp+1 , tokens 2t, 2t+1
                  af[2] = i8pair_to_h2(cd[kp], 0x4140u);   // tokens 2t+8, 2t+9
                  af[3] = i8pair_to_h2(cd[kp], 0x4342u);
                } else {
                  af[0] = e4m3pair_to_h2(ab[kp]);
                  af[1] = e4m3pair_to_h2(ab[kp] >> 16);
                  af[2] = e4m3pair_to_h2(cd[kp]);
                  af[3] = e4m3pair_to_h2(cd[kp] >> 16);
                  if (tail) { af[0] &= amask[0]; af[1] &= amask[0]; af[2] &= amask[1]; af[3] &= amask[1]; }
                }
#pragma unroll
                for (int rt = 0; rt < RT; ++rt) mma16816<MmaT>(oacc[rt][jj * 2 + kp], af, pb[rt][q][0], pb[rt][q][1]);
              }
            }
          } else {
#pragma unroll
            for (int mt = 0; mt < kKS; ++mt) {
              uint32_t af[4];
              const int tok = (lane & 7) + ((lane >> 4) << 3);
              const int dcol = 16 * mt + (((lane >> 3) & 1) << 3);
              const uint32_t addr = vbase[q] + (dcol >> 6) * (kBS * 128) + tok * 128 + ((((dcol & 63) >> 3) ^ (tok & 7)) << 4);
              // after .trans: a0 = (d 0-7, tok 0-7), a1 = (d 8-15, tok 0-7), a2 = (d 0-7, tok 8-15), a3 = (d 8-15, tok 8-15)
              ldmatrix_x4_trans(af, addr);
              if (tail) { af[0] &= amask[0]; af[1] &= amask[0]; af[2] &= amask[1]; af[3] &= amask[1]; }
#pragma unroll
              for (int rt = 0; rt < RT; ++rt) mma16816<MmaT>(oacc[rt][mt], af, pb[rt][q][0], pb[rt][q][1]);
            }
          }
        }
      }

      __syncwarp();
#pragma unroll
      for (int q = 0; q < NPI; ++q) {
        if (q < np) {
          if (lane == 0) mbar_arrive(smem_u32(&bars[kMaxStages + stg[q]]));
          stage += PG;
          if (stage >= NS) { stage -= NS; phase ^= 1u; }
        }
      }
    }
    };
    if (kI8 && fine) walk(std::bool_constant<kI8>{});
    else walk(std::false_type{});
    if (!ok) break;

    // ---- end of this CTA's part of sequence b ----
    const bool direct = PG == 1 && n_parts == 1;
    const size_t slot_row0 = (static_cast<size_t>(c + b) * PG + pgrp) * HqNq;
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      float l_row = l_run[rt];
      l_row += __shfl_xor_sync(0xffffffffu, l_row, 1);
      l_row += __shfl_xor_sync(0xffffffffu, l_row, 2);
      const float lse_row = l_row > 0.f ? m_run[rt] + log2f(l_row) - vexp : -INFINITY;
      const float inv_row = l_row > 0.f ? 1.f / l_row : 0.f;
      // accumulator columns are query rows 2t and 2t+1 of the tile
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float inv = __shfl_sync(0xffffffffu, inv_row, (2 * t + h) * 4);
        const int r = rbase + 8 * rt + 2 * t + h;
        if (r >= rows) continue;
        const int hq = kvh * a.group + r % a.group, qi = r / a.group;
        const size_t orow = (static_cast<size_t>(b) * p.Hq + hq) * p.Nq + qi;
        float* f32_row = direct ? (p.packed_f32 ? reinterpret_cast<float*>(p.out) + orow * (kD + 4) : nullptr)
                                : part_o + (slot_row0 + static_cast<size_t>(hq) * p.Nq + qi) * kD;
        uint16_t* h_row = reinterpret_cast<uint16_t*>(p.out) + orow * kD;
        auto pack = [&](float x, float y) -> uint32_t { return p.q_dtype == 0 ? pack_h2(x, y) : pack_bf2(x, y); };
        if constexpr (kQuant) {
          // 16 consecutive head-dim values: tile i holds 16g + 2i (register h) and 16g + 2i + 1 (register 2 + h)
#pragma unroll
          for (int i = 0; i < 8; i += 4) {
            const float v[8] = {oacc[rt][i][h] * inv,     oacc[rt][i][2 + h] * inv,     oacc[rt][i + 1][h] * inv, oacc[rt][i + 1][2 + h] * inv,
                                oacc[rt][i + 2][h] * inv, oacc[rt][i + 2][2 + h] * inv, oacc[rt][i + 3][h] * inv, oacc[rt][i + 3][2 + h] * inv};
            if (f32_row != nullptr) {
              float4* dst = reinterpret_cast<float4*>(f32_row + 16 * g + 2 * i);
              dst[0] = make_float4(v[0], v[1], v[2], v[3]);
              dst[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
              *reinterpret_cast<uint4*>(h_row + 16 * g + 2 * i) = make_uint4(pack(v[0], v[1]), pack(v[2], v[3]), pack(v[4], v[5]), pack(v[6], v[7]));
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < kKS; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int d = 16 * i + g + 8 * e;
              const float val = oacc[rt][i][2 * e + h] * inv;
              if (f32_row != nullptr) f32_row[d] = val;
              else if (p.q_dtype == 0) reinterpret_cast<__half*>(h_row)[d] = __float2half_rn(val);
              else reinterpret_cast<__nv_bfloat16*>(h_row)[d] = __float2bfloat16_rn(val);
            }
        }
      }
      if (t == 0 && row_of[rt] < rows) {
        const size_t orow = (static_cast<size_t>(b) * p.Hq + hq_row[rt]) * p.Nq + qi_row[rt];
        if (!direct) part_lse[slot_row0 + static_cast<size_t>(hq_row[rt]) * p.Nq + qi_row[rt]] = lse_row;
        else if (p.packed_f32) reinterpret_cast<float*>(p.out)[orow * (kD + 4) + kD] = lse_row;
        else if (p.lse != nullptr) p.lse[orow] = lse_row;
      }
    }

    u = static_cast<long long>(s0) + j_hi;
    if (u >= s1) ++b;
  }
  if (lane == 0) *status = ok ? 0 : 1;
}

// Combine of per-GPU partials: one warp per output row, lanes across the head dim.
__global__ void __launch_bounds__(256) combine_partials_kernel(const float* __restrict__ g, int R, long long rows, int D,
                                                               int out_dtype, void* __restrict__ out, float* __restrict__ lse) {
  const long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int W = D + 4;
  float m = -INFINITY;
  for (int r = 0; r < R; ++r) m = fmaxf(m, g[(static_cast<long long>(r) * rows + row) * W + D]);
  const float ms = (m == -INFINITY) ? 0.f : m;
  float wsum = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool live = lane * 4 < D;
  for (int r = 0; r < R; ++r) {
    const float* src = g + (static_cast<long long>(r) * rows + row) * W;
    const float w = exp2f(src[D] - ms);
    wsum += w;
    if (live) {
      const float4 v = *reinterpret_cast<const float4*>(src + lane * 4);
      acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
    }
  }
  const float inv = wsum > 0.f ? 1.f / wsum : 0.f;
  if (live) {
    const long long o = row * D + lane * 4;
    uint2 pk;
    if (out_dtype == 0) {
      pk = make_uint2(pack_h2(acc.x * inv, acc.y * inv), pack_h2(acc.z * inv, acc.w * inv));
      *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(out) + o) = pk;
    } else {
      pk = make_uint2(pack_bf2(acc.x * inv, acc.y * inv), pack_bf2(acc.z * inv, acc.w * inv));
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + o) = pk;
    }
  }
  if (lse != nullptr && lane == 0) lse[row] = wsum > 0.f ? m + log2f(wsum) : -INFINITY;
}

int device_sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// how a launch is cut: heads per CTA, warps per head, CTAs along the units
struct Shape {
  int hpc, row_groups, page_groups, gx;
};
Shape pick_shape(int Hkv, int rows, int num_splits) {
  Shape s;
  s.row_groups = rows > 16 ? 2 : 1;
  s.hpc = 8 / s.row_groups;
  while (Hkv % s.hpc != 0) s.hpc >>= 1;
  const int hg = Hkv / s.hpc;
  const int target = device_sm_count() * ctas_per_sm(s.hpc * s.row_groups);     // CTAs in flight over the whole grid
  s.gx = (target + hg - 1) / hg;
  if (num_splits > 0 && s.gx > num_splits) s.gx = num_splits;
  s.page_groups = 1;
  return s;
}
// int8, 8 heads to a CTA: two warps per head can take its units in turn.  At 96 registers a warp (a dozen values spilled)
// that is what keeps up with HBM (128 sequences of 512 to 32768 tokens: 785 -> 638 us), but every CTA then leaves two
// partials per sequence, which costs 3 to 6 us where there is little else (8192 tokens: 18.7 against 24.8 us); so only from
// 32 units per CTA on, as far as the longest sequence tells, and where the workspace has room for the partials.  e4m3, with
// more conversions to do at 96 registers, gains nothing (116.9 against 115.3 us).  CTAs of 4, 2 or 1 heads, two to six of
// them on an SM, are not built in that form; whether they would gain has not been measured.
bool can_take_turns(const Shape& s, int rows, int kv_dtype) { return kv_dtype == 3 && rows <= 8 && s.hpc == 8; }

template <int KV, int HPC, int D, int RT, int PG>
cudaError_t launch_t(const CUtensorMap& tmK, const CUtensorMap& tmV, const KernelArgs& a, int gx, size_t smem,
                     cudaStream_t stream) {
  auto go = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    return launch_dependent(kern, dim3(gx, a.HG), dim3((a.hpc * a.row_groups * a.page_groups + 1) * 32), smem, stream, tmK, tmV, a);
  };
  if (a.aligned) return a.inv_cap > 0.f ? go(decode_paged_kernel<KV, HPC, D, true, RT, PG, true>) : go(decode_paged_kernel<KV, HPC, D, false, RT, PG, true>);
  return a.inv_cap > 0.f ? go(decode_paged_kernel<KV, HPC, D, true, RT, PG, false>) : go(decode_paged_kernel<KV, HPC, D, false, RT, PG, false>);
}

template <int KV, int D>
cudaError_t launch_kv(const CUtensorMap& tmK, const CUtensorMap& tmV, const KernelArgs& a, int gx, size_t smem, cudaStream_t stream) {
  if (a.rows > 8) return launch_t<KV, 0, D, 2, 1>(tmK, tmV, a, gx, smem, stream);
  switch (a.hpc) {
    case 8:
      if constexpr (KV == KV_I8) {
        if (a.page_groups == 2) return launch_t<KV, 8, D, 1, 2>(tmK, tmV, a, gx, smem, stream);
      }
      return launch_t<KV, 8, D, 1, 1>(tmK, tmV, a, gx, smem, stream);
    case 4: return launch_t<KV, 4, D, 1, 1>(tmK, tmV, a, gx, smem, stream);
    case 2: return launch_t<KV, 2, D, 1, 1>(tmK, tmV, a, gx, smem, stream);
    default: return launch_t<KV, 1, D, 1, 1>(tmK, tmV, a, gx, smem, stream);
  }
}

// Warps to a row: enough that a sequence of average length has about 8 parts per warp.
template <int D>
cudaError_t launch_merge(const KernelArgs& a, int gx, cudaStream_t stream) {
  int W = 1;
  while (W < kMaxMergeWarps && static_cast<long long>(gx) * a.page_groups > 8LL * a.p.B * W) W <<= 1;
  // The successor may come in before the merge kernel has ended, but not where four or six CTAs share an SM and most of them
  // have work: they are 12 warps of 168 registers, which is all of its registers, and the next call's, placed while merge
  // blocks still run, came up one short on some SMs (presumably because those leave the four register files unevenly free)
  // and waited there for another's end.  100 sequences up to 12000 tokens, 3 queries, 2 kv heads, back to back: int8 156
  // -> 102.5 us, f16 136 -> 112; 1 kv head, 2 queries, int8 101 -> 85.5.  Elsewhere it gains up to 1 us (1 sequence of 576 tokens,
  // 2 kv heads, 4 queries 11.2 -> 10.6); a CTA without work, as far as the longest length tells, ends at once and makes room.
  // (A parameter of its own: the main kernels for 9 to 32 rows, at their limit of 168 registers, come out of the compiler
  // differently with every member of KernelArgs; one more made int8 182 -> 177 us and e4m3 186 -> 188.)
  const int let_in = ctas_per_sm(a.hpc * a.row_groups) < 4 ||
                     2 * working_ctas(static_cast<long long>(a.p.B) * ((a.p.max_kv_len + kBS - 1) / kBS), a.p.B, gx) <= gx;
  const int warps = W > kMergeWarps ? W : kMergeWarps, rows_per_block = warps / W;
  const int blocks_per_seq = (a.p.Hq * a.p.Nq + rows_per_block - 1) / rows_per_block;
  const long long blocks = static_cast<long long>(a.p.B) * blocks_per_seq;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  const size_t smem = W > 1 ? static_cast<size_t>(warps) * 32 * sizeof(float4) : 0;
  const dim3 grid(static_cast<unsigned>(blocks)), block(warps * 32);
  auto go = [&](auto kern) { return launch_dependent(kern, grid, block, smem, stream, a, gx, W, blocks_per_seq, let_in); };
  if (a.aligned) return W > 1 ? go(decode_merge_kernel<D, true, true>) : go(decode_merge_kernel<D, false, true>);
  return W > 1 ? go(decode_merge_kernel<D, true, false>) : go(decode_merge_kernel<D, false, false>);
}

}  // namespace

cudaError_t launch_combine_partials(const float* gathered, int R, long long rows, int D, int out_dtype, void* out,
                                    float* lse, cudaStream_t stream) {
  if (R <= 0 || rows <= 0) return cudaSuccess;
  const long long blocks = (rows * 32 + 255) / 256;
  combine_partials_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(gathered, R, rows, D, out_dtype, out, lse);
  return cudaGetLastError();
}

size_t decode_workspace_bytes(int B, int Hq, int Hkv, int Nq, int D, int kv_dtype, int num_splits, bool best) {
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || Nq <= 0) return 16;
  const int rows = Hq / Hkv * Nq;
  const Shape sh = pick_shape(Hkv, rows, num_splits);
  return make_layout(B, Hq, Nq, Hkv / sh.hpc, sh.gx, D, best && can_take_turns(sh, rows, kv_dtype) ? 2 : 1).total;
}

cudaError_t launch_decode_paged(const DecodeParams& p, cudaStream_t stream, char* msg, size_t msg_len) {
  const bool quant = p.kv_dtype == 3 || p.kv_dtype == 4;
  const int rows = p.Hq / p.Hkv * p.Nq;
  Shape sh = pick_shape(p.Hkv, rows, p.num_splits);
  if (can_take_turns(sh, rows, p.kv_dtype) && static_cast<long long>(p.B) * ((p.max_kv_len + kBS - 1) / kBS) >= 32LL * sh.gx &&
      p.workspace_bytes >= decode_workspace_bytes(p.B, p.Hq, p.Hkv, p.Nq, p.D, p.kv_dtype, p.num_splits, true))
    sh.page_groups = 2;
  const int hpc = sh.hpc, gx = sh.gx;
  const int HG = p.Hkv / hpc;
  const int kD = p.D;
  const int row_bytes = quant ? kD : 2 * kD;
  if (!(kD == 128 || (kD == 64 && !quant))) {
    snprintf(msg, msg_len, "head_dim %d with kv_dtype %d (built: 128 for every pool type, 64 for 16-bit pools)", kD, p.kv_dtype);
    return cudaErrorNotSupported;
  }
  if (!p.dense && (p.block_size < kBS || p.block_size % kBS != 0)) {
    snprintf(msg, msg_len, "block_size %d: pages must hold a multiple of %d tokens", p.block_size, kBS);
    return cudaErrorNotSupported;
  }

  KernelArgs a;
  a.p = p;
  a.upp = p.dense ? 1 : p.block_size / kBS;
  a.lay = make_layout(p.B, p.Hq, p.Nq, HG, gx, kD, sh.page_groups);
  a.HG = HG;
  a.group = p.Hq / p.Hkv;
  a.rows = a.group * p.Nq;
  a.hpc = hpc;
  a.row_groups = sh.row_groups;
  a.aligned = take_aligned(p.B, p.max_kv_len, gx) ? 1 : 0;
  a.page_groups = sh.page_groups;
  a.stage_kv_bytes = hpc * kBS * row_bytes;
  a.scale_bytes = quant ? kBS * p.Hkv * 2 : 0;
  a.qlo_bytes = p.kv_dtype == 3 ? hpc * sh.row_groups * sh.page_groups * (rows > 8 ? 2048 : 1024) : 0;
  const size_t per_stage = 2 * static_cast<size_t>(a.stage_kv_bytes) + 2 * static_cast<size_t>(a.scale_bytes);
  // several small CTAs share an SM when a CTA holds few heads
  const int per_sm = ctas_per_sm(hpc * sh.row_groups);
  const size_t budget = per_sm == 1 ? 200 * 1024 : (per_sm == 2 ? 100 * 1024 : (per_sm == 4 ? 50 * 1024 : 33 * 1024));
  // what a CTA takes beside its stages, the 1 KB that the hardware keeps per CTA included
  const size_t beside = 1024 + 1024 + a.qlo_bytes + 2 * kMaxStages * 8 + kMaxStages * 4 + 64 +
                        (p.B <= kSmemSeqs ? sizeof(int) * (static_cast<size_t>(p.B) + 1) : 0);
  int stages = static_cast<int>(budget / per_stage);
  if (stages > kMaxStages) stages = kMaxStages;
  // all per_sm of them at once, as the grid counts on: one stage less where the prefix sums of many sequences or the low
  // bytes of Q would be in the way
  while (stages > 2 && per_sm * (beside + stages * per_stage) > 228 * 1024) --stages;
  if (stages < 2) {
    snprintf(msg, msg_len, "Hkv=%d needs %zu bytes per stage; too large for the stage ring", p.Hkv, per_stage);
    return cudaErrorNotSupported;
  }
  a.stages = stages;
  const float sc = p.softcap > 0.f ? p.scale : p.scale * kLog2e;
  a.q_prescale = sc;
  a.cap_log2 = p.softcap * kLog2e;
  a.inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f;
  const size_t smem = beside - 1024 + static_cast<size_t>(stages) * per_stage;

  // tensor maps, in bytes: (128 B, tokens, 128-byte halves of a row, heads, batch).  A pool is one "batch" of
  // num_pages * block_size tokens with the heads of a token side by side; a dense cache has its own strides.
  CUtensorMap tmK, tmV;
  const uint32_t box[5] = {128, kBS, static_cast<uint32_t>(row_bytes / 128), static_cast<uint32_t>(hpc), 1};
  bool maps_ok;
  if (p.dense) {
    const uint64_t dims[5] = {128, static_cast<uint64_t>(p.max_kv_len), static_cast<uint64_t>(row_bytes / 128),
                              static_cast<uint64_t>(p.Hkv), static_cast<uint64_t>(p.B)};
    auto strides_of = [&](int64_t bs, int64_t hs, int64_t rs, uint64_t (&st)[4]) {
      // a size-1 dimension still needs a legal stride
      const uint64_t row = static_cast<uint64_t>(rs) * 2;
      const uint64_t head = hs > 0 ? static_cast<uint64_t>(hs) * 2 : row * p.max_kv_len;
      st[0] = row; st[1] = 128; st[2] = head;
      st[3] = bs > 0 ? static_cast<uint64_t>(bs) * 2 : head * p.Hkv;
    };
    uint64_t ks[4], vs[4];
    strides_of(p.k_bs, p.k_hs, p.k_rs, ks);
    strides_of(p.v_bs, p.v_hs, p.v_rs, vs);
    maps_ok = encode_tmap(&tmK, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, p.k_pool, dims, ks, box, CU_TENSOR_MAP_SWIZZLE_128B) &&
              encode_tmap(&tmV, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, p.v_pool, dims, vs, box, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    const uint64_t tokens = static_cast<uint64_t>(p.num_pages) * p.block_size;
    const uint64_t dims[5] = {128, tokens, static_cast<uint64_t>(row_bytes / 128), static_cast<uint64_t>(p.Hkv), 1};
    const uint64_t strides[4] = {static_cast<uint64_t>(p.Hkv) * row_bytes, 128, static_cast<uint64_t>(row_bytes),
                                 tokens * p.Hkv * row_bytes};
    maps_ok = encode_tmap(&tmK, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, p.k_pool, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B) &&
              encode_tmap(&tmV, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, p.v_pool, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  }
  if (!maps_ok) {
    snprintf(msg, msg_len, "cuTensorMapEncodeTiled failed for the K / V tensors");
    return cudaErrorInvalidValue;
  }

  unsigned char* ws = reinterpret_cast<unsigned char*>(p.workspace);
  cudaError_t e = cudaSuccess;
  if (p.B > kSmemSeqs) {
    decode_plan_kernel<<<1, 1024, 0, stream>>>(p.seq_lens, p.B, p.max_kv_len, reinterpret_cast<int*>(ws + a.lay.page_start));
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  switch (p.kv_dtype) {
    case 0: e = kD == 64 ? launch_kv<KV_F16, 64>(tmK, tmV, a, gx, smem, stream)
                            : launch_kv<KV_F16, 128>(tmK, tmV, a, gx, smem, stream); break;
    case 1: e = kD == 64 ? launch_kv<KV_BF16, 64>(tmK, tmV, a, gx, smem, stream)
                            : launch_kv<KV_BF16, 128>(tmK, tmV, a, gx, smem, stream); break;
    case 3: e = launch_kv<KV_I8, 128>(tmK, tmV, a, gx, smem, stream); break;
    case 4: e = launch_kv<KV_E4M3, 128>(tmK, tmV, a, gx, smem, stream); break;
    default: snprintf(msg, msg_len, "kv_dtype %d", p.kv_dtype); return cudaErrorNotSupported;
  }
  if (e != cudaSuccess) return e;
  return kD == 64 ? launch_merge<64>(a, gx, stream) : launch_merge<128>(a, gx, stream);
}

}  // namespace b200fa

// ---------------------------------------------------------------------------
// Decode without a caller-supplied workspace
// ---------------------------------------------------------------------------
// Scratch for b200fa_decode_paged_static: the same carve-up the workspace variant
// uses (error word, status words, page prefix sums, split partials), held in
// a fixed array that every GPU loading this library keeps until the process exits.
#define B200FA_STATIC_SCRATCH_BYTES (16u * 1024u * 1024u)
static __device__ __align__(256) unsigned char g_decode_static_scratch[B200FA_STATIC_SCRATCH_BYTES];

namespace b200fa {
void set_last_error(const char* msg);

namespace {
// In host code the array's name is only a handle; the device address has to be asked
// for, once per device, while that device is current.
cudaError_t static_scratch_address(void** out) {
  static std::mutex mu;
  static void* addr[64] = {nullptr};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
    if (e != cudaSuccess) return e;
    addr[dev] = p;
  }
  *out = addr[dev];
  return cudaSuccess;
}
}  // namespace
}  // namespace b200fa

extern "C" int32_t b200fa_decode_paged_static(const b200fa_desc* d, const void* q, const void* k_pool,
                                              const void* v_pool, const void* k_scale, const void* v_scale,
                                              const int32_t* block_table, const int32_t* seq_lens,
                                              int32_t num_pages, int32_t block_size, int32_t max_blocks,
                                              int32_t max_kv_len, void* out, float* lse, void* stream) {
  if (d == nullptr) {
    b200fa::set_last_error("descriptor is null");
    return B200FA_ERR_INVALID_ARG;
  }
  const size_t need = d->B > 0 && d->Hkv > 0 ? b200fa::decode_workspace_bytes(d->B, d->Hq, d->Hkv, d->N, d->D, d->kv_dtype, d->num_splits, false) : 16;
  if (need > B200FA_STATIC_SCRATCH_BYTES) {
    char msg[256];
    snprintf(msg, sizeof(msg),
             "b200fa_decode_paged_static: this problem needs %zu bytes of scratch, the built-in scratch holds %u; "
             "use b200fa_decode_paged with a workspace, or lower B / Hq*N",
             need, B200FA_STATIC_SCRATCH_BYTES);
    b200fa::set_last_error(msg);
    return B200FA_ERR_WORKSPACE;
  }
  void* scratch = nullptr;
  cudaError_t e = b200fa::static_scratch_address(&scratch);
  if (e != cudaSuccess) {
    char msg[256];
    snprintf(msg, sizeof(msg), "b200fa_decode_paged_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    b200fa::set_last_error(msg);
    return B200FA_ERR_CUDA;
  }
  // Same validation, planning and kernels as the workspace variant; the merge kernel
  // writes the error word at the end of every call.
  return b200fa_decode_paged(d, q, k_pool, v_pool, k_scale, v_scale, block_table, seq_lens, num_pages,
                             block_size, max_blocks, max_kv_len, out, lse, scratch,
                             B200FA_STATIC_SCRATCH_BYTES, stream);
}

// The static entry's error word sits at the start of the built-in scratch, whose address callers never see.
extern "C" int32_t b200fa_decode_paged_static_status(void* stream, int32_t* status_out) {
  if (status_out == nullptr) {
    b200fa::set_last_error("status_out is null");
    return B200FA_ERR_INVALID_ARG;
  }
  void* scratch = nullptr;
  cudaError_t e = b200fa::static_scratch_address(&scratch);
  if (e != cudaSuccess) {
    char msg[256];
    snprintf(msg, sizeof(msg), "b200fa_decode_paged_static_status: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    b200fa::set_last_error(msg);
    return B200FA_ERR_CUDA;
  }
  return b200fa_workspace_status(scratch, stream, status_out);
}
