// Page gather: pool [num_pages, block_size, H, D] -> out [B, H, max_kv_len, D].
// out[b,h,t,:] = pool[block_table[b, t / block_size], t % block_size, h, :] when
// t < seq_lens[b] and the table entry is non-negative, else zero.  A bit-exact
// copy with 64-bit offsets; same contract as the reference's paged_kv_gather
// (csrc/mfa_paged_gather.cpp:44-80 kernel, 89-129 CPU loop).
#include <cuda_fp8.h>

#include "common.cuh"
#include "launch.h"

namespace b200fa {

namespace {

// I: index type of the flattened chunk space (32-bit whenever it fits: the index is split by run-time divisors per chunk)
template <typename I>
__global__ void __launch_bounds__(256) paged_kv_gather_kernel(
    const uint4* __restrict__ pool, const int32_t* __restrict__ block_table,
    const int32_t* __restrict__ seq_lens, int H, int chunks_per_row /* D*elem_bytes/16 */,
    int block_size, int max_blocks, int max_kv_len, long long total_chunks, uint4* __restrict__ out) {
  const I stride = static_cast<I>(gridDim.x) * blockDim.x, total = static_cast<I>(total_chunks);
  for (I idx = static_cast<I>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    // idx = ((b*H + h)*max_kv_len + t)*chunks_per_row + c
    const int c = static_cast<int>(idx % static_cast<I>(chunks_per_row));
    I rem = idx / static_cast<I>(chunks_per_row);
    const int t = static_cast<int>(rem % static_cast<I>(max_kv_len));
    rem /= static_cast<I>(max_kv_len);
    const int h = static_cast<int>(rem % static_cast<I>(H));
    const int b = static_cast<int>(rem / static_cast<I>(H));
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (t < seq_lens[b]) {
      const int page = block_table[static_cast<long long>(b) * max_blocks + t / block_size];
      if (page >= 0) {
        const long long src =
            ((static_cast<long long>(page) * block_size + (t % block_size)) * H + h) * chunks_per_row + c;
        val = pool[src];
      }
    }
    out[idx] = val;
  }
}

// Gather + dequantise: one thread per 16 pool bytes (16 values of one (token, head) row), written as 32 bytes of the
// 16-bit output.  value = T(float(x) * float(scale)): one rounding, to the output type, as the host definition has it.
template <typename T, bool E4M3>
__global__ void __launch_bounds__(256) paged_kv_gather_dequant_kernel(
    const uint4* __restrict__ pool, const __half* __restrict__ scale, const int32_t* __restrict__ block_table,
    const int32_t* __restrict__ seq_lens, int H, int chunks_per_row /* D / 16 */, int block_size, int max_blocks,
    int max_kv_len, long long total_chunks, uint4* __restrict__ out) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total_chunks; idx += stride) {
    const int c = static_cast<int>(idx % chunks_per_row);
    long long rem = idx / chunks_per_row;
    const int t = static_cast<int>(rem % max_kv_len);
    rem /= max_kv_len;
    const int h = static_cast<int>(rem % H);
    const int b = static_cast<int>(rem / H);
    uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
    if (t < seq_lens[b]) {
      const int page = block_table[static_cast<long long>(b) * max_blocks + t / block_size];
      if (page >= 0) {
        const long long rowi = (static_cast<long long>(page) * block_size + (t % block_size)) * H + h;
        const uint4 raw = pool[rowi * chunks_per_row + c];
        const float sc = __half2float(scale[rowi]);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t byte = (w[i] >> (8 * e)) & 0xffu;
            if (E4M3) {
              const __half_raw hr = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3);
              f[e] = __half2float(__half(hr));
            } else {
              f[e] = static_cast<float>(static_cast<int>(static_cast<signed char>(byte)));
            }
          }
          o[2 * i] = Elem<T>::pack(f[0] * sc, f[1] * sc);
          o[2 * i + 1] = Elem<T>::pack(f[2] * sc, f[3] * sc);
        }
        lo = make_uint4(o[0], o[1], o[2], o[3]);
        hi = make_uint4(o[4], o[5], o[6], o[7]);
      }
    }
    out[2 * idx] = lo;
    out[2 * idx + 1] = hi;
  }
}

// The same for K and V in one launch, for the forward over per-sequence key counts (blockIdx.y: 0 = K, 1 = V): rows up to
// the end of a sequence's last 64-key tile are written (zeros beyond its length, for the tensor core multiplies them all
// the same), the rest of the padded output is not, since nothing reads it.  Bound by HBM: 386 bytes per token and head.  A
// block takes kDqTokens tokens of one sequence and all heads, a thread 16 values at a time, four in flight; whole blocks
// beyond a sequence leave at once.  4 sequences of 1000 to 8000 tokens, 8 heads, int8: two launches over the padded
// shape, a chain of 64-bit divisions per 16 values, took 40 us.
constexpr int kDqTokens = 32;
constexpr int kKeyTile = 64;      // keys per tile of the forward kernel

template <typename T, bool E4M3>
__global__ void __launch_bounds__(256) paged_kv_dequant_pair_kernel(
    const uint4* __restrict__ k_pool, const uint4* __restrict__ v_pool, const __half* __restrict__ k_scale,
    const __half* __restrict__ v_scale, const int32_t* __restrict__ block_table, const int32_t* __restrict__ seq_lens, int H,
    unsigned cpr, int block_size, int max_blocks, int max_kv_len, int num_pages, int tiles, uint4* __restrict__ k_out,
    uint4* __restrict__ v_out) {
  __shared__ int s_row[kDqTokens];       // token's row in the pool, -1: zeros
  const int b = blockIdx.x / tiles, t0 = (blockIdx.x % tiles) * kDqTokens;
  const int len = min(max(seq_lens[b], 0), max_kv_len);
  const int end = min((len + kKeyTile - 1) / kKeyTile * kKeyTile, max_kv_len);
  if (t0 >= end) return;
  const uint4* pool = blockIdx.y == 0 ? k_pool : v_pool;
  const __half* scale = blockIdx.y == 0 ? k_scale : v_scale;
  uint4* out = blockIdx.y == 0 ? k_out : v_out;
  if (threadIdx.x < kDqTokens) {
    const int t = t0 + threadIdx.x;
    int row = -1;
    if (t < len) {
      const int page = block_table[static_cast<long long>(b) * max_blocks + t / block_size];
      if (page >= 0 && page < num_pages) row = page * block_size + t % block_size;
    }
    s_row[threadIdx.x] = row;
  }
  __syncthreads();
  const unsigned per_head = kDqTokens * cpr, total = per_head * H;
  constexpr int kFlight = 4;
  for (unsigned i0 = threadIdx.x; i0 < total; i0 += 256 * kFlight) {
    uint4 raw[kFlight];
    float sc[kFlight];
    long long dst[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
      const unsigned i = i0 + 256 * k;
      raw[k] = make_uint4(0u, 0u, 0u, 0u);
      sc[k] = 0.f;
      dst[k] = -1;
      if (i < total) {
        const unsigned h = i / per_head, r = i % per_head, t = r / cpr, c = r % cpr;
        if (static_cast<int>(t0 + t) < end) {
          dst[k] = ((static_cast<long long>(b) * H + h) * max_kv_len + t0 + t) * cpr + c;
          const int row = s_row[t];
          if (row >= 0) {
            const long long src = static_cast<long long>(row) * H + h;
            raw[k] = __ldg(pool + src * cpr + c);
            sc[k] = __half2float(scale[src]);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
      if (dst[k] < 0) continue;
      const uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
      uint32_t o[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t byte = (w[q] >> (8 * e)) & 0xffu;
          if (E4M3) {
            const __half_raw hr = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3);
            f[e] = __half2float(__half(hr));
          } else {
            f[e] = static_cast<float>(static_cast<int>(static_cast<signed char>(byte)));
          }
        }
        o[2 * q] = Elem<T>::pack(f[0] * sc[k], f[1] * sc[k]);
        o[2 * q + 1] = Elem<T>::pack(f[2] * sc[k], f[3] * sc[k]);
      }
      out[2 * dst[k]] = make_uint4(o[0], o[1], o[2], o[3]);
      out[2 * dst[k] + 1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  }
}

// The transpose of the gather, for gradients: grad_pool[page, t % bs, h, :] += grad[b, h, t, :] for t < seq_lens[b]
// and a non-negative table entry (the role of _scatter_to_pool, mlx_mfa/attention.py:2878-2940).  The pool-shaped
// output must start at zero; a page listed by several sequences (a shared prefix) accumulates all of them, which is
// why the adds are packed 16-bit atomics rather than stores.
template <typename T2>
__global__ void __launch_bounds__(256) paged_kv_scatter_add_kernel(
    const uint4* __restrict__ grad, const int32_t* __restrict__ block_table, const int32_t* __restrict__ seq_lens, int H,
    int chunks_per_row, int block_size, int max_blocks, int max_kv_len, long long total_chunks, T2* __restrict__ grad_pool) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total_chunks; idx += stride) {
    const int c = static_cast<int>(idx % chunks_per_row);
    long long rem = idx / chunks_per_row;
    const int t = static_cast<int>(rem % max_kv_len);
    rem /= max_kv_len;
    const int h = static_cast<int>(rem % H);
    const int b = static_cast<int>(rem / H);
    if (t >= seq_lens[b]) continue;
    const int page = block_table[static_cast<long long>(b) * max_blocks + t / block_size];
    if (page < 0) continue;
    const uint4 v = grad[idx];
    const long long dst = (((static_cast<long long>(page) * block_size + (t % block_size)) * H + h) * chunks_per_row + c) * 4;
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) atomicAdd(grad_pool + dst + i, *reinterpret_cast<const T2*>(&w[i]));
  }
}

}  // namespace

cudaError_t launch_paged_scatter_add(const void* grad, const int32_t* block_table, const int32_t* seq_lens, int B, int H,
                                     int D, int dtype, int block_size, int max_blocks, int max_kv_len, void* grad_pool,
                                     cudaStream_t stream) {
  const int cpr = D * 2 / 16;
  const long long total = static_cast<long long>(B) * H * max_kv_len * cpr;
  if (total == 0) return cudaSuccess;
  long long blocks = (total + 255) / 256;
  const long long cap = 148LL * 32;
  if (blocks > cap) blocks = cap;
  if (dtype == 0)
    paged_kv_scatter_add_kernel<__half2><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        reinterpret_cast<const uint4*>(grad), block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total,
        reinterpret_cast<__half2*>(grad_pool));
  else
    paged_kv_scatter_add_kernel<__nv_bfloat162><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        reinterpret_cast<const uint4*>(grad), block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total,
        reinterpret_cast<__nv_bfloat162*>(grad_pool));
  return cudaGetLastError();
}

cudaError_t launch_paged_gather_dequant(const void* pool, const void* scale, const int32_t* block_table,
                                        const int32_t* seq_lens, int B, int H, int D, int pool_dtype, int out_dtype,
                                        int block_size, int max_blocks, int max_kv_len, void* out, cudaStream_t stream) {
  const int cpr = D / 16;
  const long long total = static_cast<long long>(B) * H * max_kv_len * cpr;
  if (total == 0) return cudaSuccess;
  long long blocks = (total + 255) / 256;
  const long long cap = 148LL * 32;
  if (blocks > cap) blocks = cap;
  const unsigned g = static_cast<unsigned>(blocks);
  const uint4* pl = reinterpret_cast<const uint4*>(pool);
  const __half* sc = reinterpret_cast<const __half*>(scale);
  uint4* o = reinterpret_cast<uint4*>(out);
  const bool e4 = pool_dtype == 4;
  if (out_dtype == 0) {
    if (e4) paged_kv_gather_dequant_kernel<__half, true><<<g, 256, 0, stream>>>(pl, sc, block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total, o);
    else paged_kv_gather_dequant_kernel<__half, false><<<g, 256, 0, stream>>>(pl, sc, block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total, o);
  } else {
    if (e4) paged_kv_gather_dequant_kernel<__nv_bfloat16, true><<<g, 256, 0, stream>>>(pl, sc, block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total, o);
    else paged_kv_gather_dequant_kernel<__nv_bfloat16, false><<<g, 256, 0, stream>>>(pl, sc, block_table, seq_lens, H, cpr, block_size, max_blocks, max_kv_len, total, o);
  }
  return cudaGetLastError();
}

cudaError_t launch_paged_dequant_pair(const void* k_pool, const void* v_pool, const void* k_scale, const void* v_scale,
                                      const int32_t* block_table, const int32_t* seq_lens, int B, int H, int D, int pool_dtype,
                                      int out_dtype, int num_pages, int block_size, int max_blocks, int max_kv_len, void* k_out,
                                      void* v_out, cudaStream_t stream) {
  if (B <= 0 || max_kv_len <= 0) return cudaSuccess;
  const int tiles = static_cast<int>((static_cast<long long>(max_kv_len) + kDqTokens - 1) / kDqTokens);
  const dim3 grid(static_cast<unsigned>(tiles) * B, 2);
  auto go = [&](auto kern) {
    kern<<<grid, 256, 0, stream>>>(static_cast<const uint4*>(k_pool), static_cast<const uint4*>(v_pool),
                                   static_cast<const __half*>(k_scale), static_cast<const __half*>(v_scale), block_table, seq_lens, H,
                                   static_cast<unsigned>(D / 16), block_size, max_blocks, max_kv_len, num_pages, tiles,
                                   static_cast<uint4*>(k_out), static_cast<uint4*>(v_out));
  };
  if (out_dtype == 0) {
    if (pool_dtype == 4) go(paged_kv_dequant_pair_kernel<__half, true>); else go(paged_kv_dequant_pair_kernel<__half, false>);
  } else {
    if (pool_dtype == 4) go(paged_kv_dequant_pair_kernel<__nv_bfloat16, true>); else go(paged_kv_dequant_pair_kernel<__nv_bfloat16, false>);
  }
  return cudaGetLastError();
}

cudaError_t launch_paged_gather(const void* pool, const int32_t* block_table, const int32_t* seq_lens,
                                int B, int H, int D, int elem_bytes, int block_size, int max_blocks,
                                int max_kv_len, void* out, cudaStream_t stream) {
  const int cpr = D * elem_bytes / 16;
  const long long total = static_cast<long long>(B) * H * max_kv_len * cpr;
  if (total == 0) return cudaSuccess;
  long long blocks = (total + 255) / 256;
  const long long cap = 148LL * 32;
  if (blocks > cap) blocks = cap;
  if (total < (1LL << 31))
    paged_kv_gather_kernel<uint32_t><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        reinterpret_cast<const uint4*>(pool), block_table, seq_lens, H, cpr, block_size, max_blocks,
        max_kv_len, total, reinterpret_cast<uint4*>(out));
  else
    paged_kv_gather_kernel<long long><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        reinterpret_cast<const uint4*>(pool), block_table, seq_lens, H, cpr, block_size, max_blocks,
        max_kv_len, total, reinterpret_cast<uint4*>(out));
  return cudaGetLastError();
}

}  // namespace b200fa
