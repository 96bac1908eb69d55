// float32 forward kernel: FFMA on the CUDA cores with fp32 accumulation and
// precise exp2f/tanhf, for the <= 1e-5 parity bar that tf32 tensor-core inputs
// (10-bit mantissa) cannot meet.  Fills the role of the reference's fp32 forward
// (csrc/mfa_attention.cpp:85-129, generator csrc/mfa_shader_gen.cpp:105-303).
// Same masks, softcap order and lse convention as the 16-bit kernels.
//
// Bound by the FMA pipe: a 64 x 64 tile at head_dim 128 is 2 * 64 * 64 * 128 FMAs, 8192 clk of an SM.  What it takes:
//   * registers: a thread holds 8 x 4 scores and 8 x 8 output values, so 12 (16) 16-byte shared loads feed 128 (256)
//     FMAs and shared memory is half idle.  With 4 x 4 and 4 x 8 per thread a tile took 18000 clk.
//   * two CTAs of four warps per SM, one loading while the other computes; P lies over K to make room for both.
//   * equal shares: the units (query tile, key tile) of all heads form one list, and CTA c of G takes the units
//     [c U / G, (c + 1) U / G), two CTAs per SM, whatever the mask leaves of each query tile.  A query tile that two or
//     more CTAs share leaves partials (O, row max, row sum), which fwd_f32_merge_kernel adds up.  With one CTA per query
//     tile the longest row of tiles set the time: 16 tiles on a causal N = 1024 where an SM's share is 7.4.
// B = 1, H = 8, N = 1024, D = 128, causal: 153 -> 72 us.
#include "common.cuh"
#include "launch.h"

namespace b200fa {

namespace {

constexpr int kBQ = 64;
constexpr int kBK = 64;
constexpr int kThreads = 128;
constexpr int kCtasPerSm = 2;
constexpr int kPad = 4;  // floats; makes 16-byte reads of consecutive rows conflict-free
constexpr int kLDP = kBK + kPad;

struct F32Args {
  FwdParams p;
  int n_qt;                  // query tiles per (batch | sequence, head)
  long long units_per_head;  // split launches: units of one head's query tiles
  long long units;           // ... of all heads
  float* part_ml;            // [2 G][64][2] row max, row sum (base 2); null = one CTA per query tile
  float* part_o;             // [2 G][64][D], not normalised
};

// key tiles [begin, end) of query tile qt; a tile without any (blind) keeps one unit, which is masked throughout
struct KeyTiles {
  int begin, end;
  bool blind;
};
__host__ __device__ inline KeyTiles key_tiles(int qt, int N, int S, int causal, int window_left) {
  const int q0 = qt * kBQ, off = S - N;
  int k_hi = S;
  if (causal && q0 + kBQ + off < S) k_hi = q0 + kBQ + off;
  int k_lo = 0;
  if (window_left >= 0 && q0 + off - window_left > 0) k_lo = q0 + off - window_left;
  KeyTiles t;
  t.begin = k_lo / kBK;
  t.end = k_hi > 0 ? (k_hi + kBK - 1) / kBK : 0;
  t.blind = t.end <= t.begin;
  if (t.blind) t.end = t.begin + 1;
  return t;
}

template <int D, int LD>
__device__ __forceinline__ void load_rows(float* s, const float* g, int64_t rs, int row0, int limit, int tid) {
  constexpr int CH = D / 4;
  const uint32_t base = smem_u32(s);
#pragma unroll 8
  for (int i = tid; i < 64 * CH; i += kThreads) {
    const int r = i / CH, c = i % CH;
    const bool in = row0 + r < limit;
    cp_async16(base + (r * LD + c * 4) * 4, g + (in ? static_cast<int64_t>(row0 + r) * rs : 0) + c * 4, in);
  }
}

// first query tile whose units end beyond u (u < units of the head); *u becomes the position inside it.  One warp.
__device__ __forceinline__ int find_tile(long long* u, const F32Args& a, int lane) {
  const FwdParams& p = a.p;
  for (int base = 0;; base += 32) {
    const int qt = base + lane;
    const KeyTiles t = key_tiles(qt < a.n_qt ? qt : a.n_qt - 1, p.N, p.S, p.causal, p.window_left);
    const int n = qt < a.n_qt ? t.end - t.begin : 0;
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const unsigned beyond = __ballot_sync(0xffffffffu, x > *u);
    if (beyond != 0u || base + 32 >= a.n_qt) {
      const int l = beyond != 0u ? __ffs(beyond) - 1 : (a.n_qt - 1 - base);
      *u -= __shfl_sync(0xffffffffu, x - n, l);
      return base + l;
    }
    *u -= __shfl_sync(0xffffffffu, x, 31);
  }
}

template <int D, bool VARLEN>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) fa_fwd_f32_kernel(const F32Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = D + kPad;
  constexpr int NC = D / 64;  // float4 output columns per thread
  float* sQ = reinterpret_cast<float*>(smem_raw);
  float* sK = sQ + kBQ * LD;
  float* sP = sK;             // P takes K's place once the scores are made
  float* sV = sK + kBK * LD;
  const FwdParams& p = a.p;

  const int tid = threadIdx.x, lane = tid & 31;
  const int ty = tid >> 4, tx = tid & 15;       // rows ty + 8 i, score columns tx + 16 j, output columns 4 tx + 64 c
  const bool split = a.part_ml != nullptr;
  pdl_launch_dependents();

  // this CTA's first query tile, the place in its key tiles, and how many units it takes
  int bh, qt, at;
  long long left;
  if (split) {
    const long long lo = blockIdx.x * a.units / gridDim.x, hi = (blockIdx.x + 1LL) * a.units / gridDim.x;
    left = hi - lo;
    bh = static_cast<int>(lo / a.units_per_head);
    long long u = lo - bh * a.units_per_head;
    qt = find_tile(&u, a, lane);
    at = static_cast<int>(u);
  } else {
    bh = blockIdx.z * p.Hq + blockIdx.y;
    qt = a.n_qt - 1 - static_cast<int>(blockIdx.x);       // the longest ones of a causal mask first
    at = 0;
    left = 0x7fffffff;
  }

  for (int seg = 0; left > 0; ++seg) {
    const int head = bh % p.Hq;
    const int kvh = head / p.gqa;
    int bb = bh / p.Hq;
    int q_begin = 0, k_begin = 0, N = p.N, S = p.S;
    if (VARLEN) {
      q_begin = p.cu_q[bb];
      N = p.cu_q[bb + 1] - q_begin;
      k_begin = p.cu_k[bb];
      S = p.cu_k[bb + 1] - k_begin;
      bb = 0;
    }
    const int q0 = qt * kBQ;
    if (q0 >= N) return;
    const int off = S - N;
    const KeyTiles kts = key_tiles(qt, N, S, p.causal, p.window_left);
    const int kt_begin = kts.begin + at;
    const int kt_end = static_cast<int>(min(static_cast<long long>(kts.end), kt_begin + left));
    const int S_read = kts.blind ? 0 : S;        // what no row sees is not read: 0 * inf would be NaN
    const bool whole = at == 0 && kt_end == kts.end;

    const float* qg = reinterpret_cast<const float*>(p.q) + bb * p.q_bs + head * p.q_hs + q_begin * p.q_rs;
    const float* kg = reinterpret_cast<const float*>(p.k) + bb * p.k_bs + kvh * p.k_hs + k_begin * p.k_rs;
    const float* vg = reinterpret_cast<const float*>(p.v) + bb * p.v_bs + kvh * p.v_hs + k_begin * p.v_rs;
    float* og = reinterpret_cast<float*>(p.o) + bb * p.o_bs + head * p.o_hs + q_begin * p.o_rs;

    float4 o[8][NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < NC; ++c) o[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    float row_max[8], row_sum[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { row_max[i] = -INFINITY; row_sum[i] = 0.f; }

    __syncthreads();  // the previous segment has read Q
    load_rows<D, LD>(sQ, qg, p.q_rs, q0, N, tid);

    const bool use_cap = p.softcap > 0.f;
    const float alibi = p.alibi != nullptr ? p.alibi[head] : 0.f;

    for (int kt = kt_begin; kt < kt_end; ++kt) {
      const int k0 = kt * kBK;
      __syncthreads();  // previous tile fully consumed
      load_rows<D, LD>(sK, kg, p.k_rs, k0, S_read, tid);
      cp_async_commit();                       // Q (first tile) and K
      load_rows<D, D>(sV, vg, p.v_rs, k0, S_read, tid);
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();

      float acc[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 2
      for (int d = 0; d < D; d += 4) {
        float4 q4[8], k4[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) q4[i] = *reinterpret_cast<const float4*>(sQ + (ty + 8 * i) * LD + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(sK + (tx + 16 * j) * LD + d);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j] = fmaf(q4[i].x, k4[j].x, acc[i][j]);
            acc[i][j] = fmaf(q4[i].y, k4[j].y, acc[i][j]);
            acc[i][j] = fmaf(q4[i].z, k4[j].z, acc[i][j]);
            acc[i][j] = fmaf(q4[i].w, k4[j].w, acc[i][j]);
          }
      }

      // scale, softcap, masks; scores move to the base-2 domain
      const bool edge = k0 + kBK > S || (p.causal && k0 + kBK - 1 > q0 + off) || (p.window_left >= 0 && k0 < q0 + kBQ - 1 + off - p.window_left);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = q0 + ty + 8 * i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = k0 + tx + 16 * j;
          float sc = acc[i][j] * p.scale;
          if (use_cap) sc = tanhf(sc / p.softcap) * p.softcap;
          if (p.alibi != nullptr) sc = fmaf(alibi, static_cast<float>(col - (row + off)), sc);
          sc *= kLog2e;
          if (edge) {
            bool vis = col < S;
            if (p.causal) vis = vis && (col <= row + off);
            if (p.window_left >= 0) vis = vis && (col >= row + off - p.window_left);
            if (!vis) sc = -INFINITY;
          }
          acc[i][j] = sc;
        }
      }

      __syncthreads();  // K is read: P may be written over it
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float mx = fmaxf(fmaxf(acc[i][0], acc[i][1]), fmaxf(acc[i][2], acc[i][3]));
#pragma unroll
        for (int sft = 1; sft < 16; sft <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sft));
        mx = fmaxf(mx, row_max[i]);
        const float msub = (mx == -INFINITY) ? 0.f : mx;
        const float corr = exp2f(row_max[i] - msub);
        row_max[i] = mx;
        row_sum[i] *= corr;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          o[i][c].x *= corr; o[i][c].y *= corr; o[i][c].z *= corr; o[i][c].w *= corr;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float pv = exp2f(acc[i][j] - msub);
          row_sum[i] += pv;
          sP[(ty + 8 * i) * kLDP + tx + 16 * j] = pv;
        }
      }
      cp_async_wait<0>();
      __syncthreads();  // V has landed for every thread (a row of P is read by the 16 lanes that wrote it)

      // O += P V
#pragma unroll 2
      for (int key = 0; key < kBK; key += 4) {
        float4 p4[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p4[i] = *reinterpret_cast<const float4*>(sP + (ty + 8 * i) * kLDP + key);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          float4 v4[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) v4[c] = *reinterpret_cast<const float4*>(sV + (key + kk) * D + tx * 4 + 64 * c);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float pv = kk == 0 ? p4[i].x : kk == 1 ? p4[i].y : kk == 2 ? p4[i].z : p4[i].w;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              o[i][c].x = fmaf(pv, v4[c].x, o[i][c].x);
              o[i][c].y = fmaf(pv, v4[c].y, o[i][c].y);
              o[i][c].z = fmaf(pv, v4[c].z, o[i][c].z);
              o[i][c].w = fmaf(pv, v4[c].w, o[i][c].w);
            }
          }
        }
      }
    }

    // the slot of a partial: 2 c for the CTA's first segment, 2 c + 1 for a later one (which can only be its last)
    const size_t slot = (2 * static_cast<size_t>(blockIdx.x) + (seg > 0 ? 1 : 0)) * kBQ;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float sum = row_sum[i];
#pragma unroll
      for (int sft = 1; sft < 16; sft <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sft);
      const int r = ty + 8 * i, row = q0 + r;
      if (row >= N) continue;
      if (!whole) {
#pragma unroll
        for (int c = 0; c < NC; ++c) *reinterpret_cast<float4*>(a.part_o + (slot + r) * D + tx * 4 + 64 * c) = o[i][c];
        if (tx == 0) *reinterpret_cast<float2*>(a.part_ml + (slot + r) * 2) = make_float2(row_max[i], sum);
        continue;
      }
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float4 val = o[i][c];
        val.x *= inv; val.y *= inv; val.z *= inv; val.w *= inv;
        *reinterpret_cast<float4*>(og + static_cast<int64_t>(row) * p.o_rs + tx * 4 + 64 * c) = val;
      }
      if (p.lse != nullptr && tx == 0) {
        float* lg = p.lse + bb * p.lse_bs + head * p.lse_hs + q_begin;
        lg[row] = sum > 0.f ? row_max[i] + log2f(sum) : -INFINITY;
      }
    }

    if (!split) return;
    left -= kt_end - kt_begin;
    at = 0;
    if (++qt == a.n_qt) { qt = 0; ++bh; }
  }
}

// Sum of the partials of every query tile that two or more CTAs of the split launch shared: one warp per row, lanes along
// the head dim, eight blocks to a query tile.  Bound by latency: a row is two dependent reads, so a warp has one (one block
// per query tile, eight rows per warp in turn: 19.7 us at B = 1, H = 8, N = 1024).  The tiles that one CTA finished cost a
// look at the shares.
constexpr int kMergeWarps = 8;
template <int D>
__global__ void __launch_bounds__(kMergeWarps * 32) fwd_f32_merge_kernel(const F32Args a, int G) {
  const FwdParams& p = a.p;
  const int bh = blockIdx.x / a.n_qt, qt = blockIdx.x % a.n_qt;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // units before this query tile
  long long u0 = 0;
  for (int i = lane; i < qt; i += 32) {
    const KeyTiles t = key_tiles(i, p.N, p.S, p.causal, p.window_left);
    u0 += t.end - t.begin;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) u0 += __shfl_xor_sync(0xffffffffu, u0, s);
  u0 += bh * a.units_per_head;
  const KeyTiles t = key_tiles(qt, p.N, p.S, p.causal, p.window_left);
  const long long u1 = u0 + (t.end - t.begin) - 1;
  const int c0 = static_cast<int>(((u0 + 1) * G - 1) / a.units), c1 = static_cast<int>(((u1 + 1) * G - 1) / a.units);
  pdl_wait();
  if (c0 == c1) return;
  const int first = 2 * c0 + (c0 * a.units / G < u0 ? 1 : 0);      // slot of the first part; those of the others are even
  const int head = bh % p.Hq, bb = bh / p.Hq;
  const bool live = lane * 4 < D;
  const int r = blockIdx.y * kMergeWarps + warp;
  if (qt * kBQ + r < p.N) {
    float m = -INFINITY;
#pragma unroll 4
    for (int c = c0; c <= c1; ++c) m = fmaxf(m, a.part_ml[(static_cast<size_t>(c == c0 ? first : 2 * c) * kBQ + r) * 2]);
    const float ms = (m == -INFINITY) ? 0.f : m;
    float sum = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int c = c0; c <= c1; ++c) {
      const size_t at = static_cast<size_t>(c == c0 ? first : 2 * c) * kBQ + r;
      const float2 ml = *reinterpret_cast<const float2*>(a.part_ml + at * 2);
      const float w = exp2f(ml.x - ms);
      sum = fmaf(w, ml.y, sum);
      if (live) {
        const float4 v = *reinterpret_cast<const float4*>(a.part_o + at * D + lane * 4);
        acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
      }
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    const int row = qt * kBQ + r;
    if (live)
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.o) + bb * p.o_bs + head * p.o_hs + static_cast<int64_t>(row) * p.o_rs + lane * 4) =
          make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    if (p.lse != nullptr && lane == 0)
      p.lse[bb * p.lse_bs + head * p.lse_hs + row] = sum > 0.f ? m + log2f(sum) : -INFINITY;
  }
}

// CTAs of a split launch, and its units
struct Split {
  int G;
  long long units_per_head, units;
};
Split plan_split(int B, int Hq, int N, int S, int causal, int window_left, int sm_count) {
  Split s = {0, 0, 0};
  const int n_qt = (N + kBQ - 1) / kBQ;
  for (int i = 0; i < n_qt; ++i) {
    const KeyTiles t = key_tiles(i, N, S, causal, window_left);
    s.units_per_head += t.end - t.begin;
  }
  s.units = s.units_per_head * B * Hq;
  const long long want = static_cast<long long>(kCtasPerSm) * sm_count;
  s.G = static_cast<int>(s.units < want ? s.units : want);
  return s;
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  return n;
}

template <int D, bool VARLEN>
cudaError_t launch_one(const FwdParams& p, int nbatch, int max_q, void* workspace, cudaStream_t stream) {
  constexpr size_t smem = (static_cast<size_t>(2) * 64 * (D + kPad) + 64 * D) * sizeof(float);
  static_assert(64 * kLDP <= 64 * (D + kPad), "P lies over K");
  auto kern = fa_fwd_f32_kernel<D, VARLEN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  F32Args a = {};
  a.p = p;
  a.n_qt = (max_q + kBQ - 1) / kBQ;
  if (VARLEN || workspace == nullptr) {
    kern<<<dim3(a.n_qt, p.Hq, nbatch), kThreads, smem, stream>>>(a);
    return cudaGetLastError();
  }
  const Split s = plan_split(p.B, p.Hq, p.N, p.S, p.causal, p.window_left, sm_count());
  a.units_per_head = s.units_per_head;
  a.units = s.units;
  a.part_o = reinterpret_cast<float*>(workspace);
  a.part_ml = a.part_o + static_cast<size_t>(2) * s.G * kBQ * D;
  kern<<<s.G, kThreads, smem, stream>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(a.n_qt) * p.Hq * p.B, kBQ / kMergeWarps);
  cfg.blockDim = dim3(kMergeWarps * 32);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fwd_f32_merge_kernel<D>, a, s.G);
}

}  // namespace

size_t fwd_f32_workspace_bytes(int B, int Hq, int N, int S, int D, int causal, int window_left) {
  if (B <= 0 || Hq <= 0 || N <= 0) return 0;
  const long long tiles = static_cast<long long>((N + kBQ - 1) / kBQ) * Hq * B;
  if (tiles > 0x7fffffffLL) return 0;
  const Split s = plan_split(B, Hq, N, S, causal, window_left, sm_count());
  return static_cast<size_t>(2) * s.G * kBQ * (D + 2) * sizeof(float);
}

cudaError_t launch_fwd_f32(const FwdParams& p, int D, bool varlen, int nbatch, int max_q, void* workspace,
                           cudaStream_t stream) {
  if (max_q <= 0 || nbatch <= 0) return cudaSuccess;
  if (D == 64) return varlen ? launch_one<64, true>(p, nbatch, max_q, nullptr, stream)
                             : launch_one<64, false>(p, nbatch, max_q, workspace, stream);
  if (D == 128) return varlen ? launch_one<128, true>(p, nbatch, max_q, nullptr, stream)
                              : launch_one<128, false>(p, nbatch, max_q, workspace, stream);
  return cudaErrorInvalidValue;
}

}  // namespace b200fa
