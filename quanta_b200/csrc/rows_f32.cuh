// Products of a few float32 rows with a float32 matrix [rows of weights, K] that is read once.
//
// Bound by the weights' bytes.  A warp owns FW rows of weights and reads each of them from end to end, 16 bytes a lane, U
// steps ahead (2 or 4 KB in flight a warp; 148 SMs need some 35 KB each for the whole bandwidth); the few input rows come
// out of L1.  A result is 32 lanes' partial sums added in one tree (lanes 16, 8, 4, 2, 1 apart), so a row's value depends on
// K alone, not on how many rows or which weights share the launch.
#pragma once
#include "common.cuh"

__device__ __forceinline__ float4 qb_ldg_stream(const float* p) {      // read once: not kept in L1, which the inputs use
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Rows of inputs for a block's products: copied to shared memory when they fit (every step of a warp reads all of them, and a
// block's warps would each wait for the same L2 lines step after step: 4 rows of 2,048 x 3,072 10.0 us without the copy, 8.4 with it), else read where they lie.
constexpr int QB_ROWS_SMEM = 96 * 1024;

__host__ __device__ __forceinline__ int qb_rows_smem(int rows, int K) {       // bytes of the copy, 0: none
  const long long n = (long long)rows * K * (long long)sizeof(float);
  return n <= QB_ROWS_SMEM ? (int)n : 0;
}

// Starts the copy of `rows` rows (row r at src(r)) by all threads of the block; qb_rows_ready waits for it.
template <typename Src>
__device__ __forceinline__ void qb_rows_copy(float* dst, Src src, int rows, int K) {
  const int pieces = K >> 2;
  for (int r = 0; r < rows; ++r) {
    const float* from = src(r);
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + (size_t)r * K + 4 * i);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from + 4 * i) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void qb_rows_ready() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

// acc[f][r] = this lane's part of w[f] . x_r, where x(r, k) gives four values of input row r; K is a multiple of 4, the weights'
// rows start on 16 bytes.  `ready` is called once the first weights are on their way.
template <int FW, int R, int U, typename X, typename Ready>
__device__ __forceinline__ void qb_rows_dot(const float* const (&w)[FW], X x, Ready ready, int K, int lane, float (&acc)[FW][R]) {
#pragma unroll
  for (int f = 0; f < FW; ++f)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[f][r] = 0.f;
  float4 buf[U][FW];
  auto fetch = [&](int k, float4 (&b)[FW]) {
#pragma unroll
    for (int f = 0; f < FW; ++f) b[f] = k < K ? qb_ldg_stream(w[f] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
#pragma unroll
  for (int u = 0; u < U; ++u) fetch(lane * 4 + u * 128, buf[u]);
  ready();
  for (int k0 = lane * 4; k0 < K; k0 += 128 * U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * 128;
      float4 now[FW];
#pragma unroll
      for (int f = 0; f < FW; ++f) now[f] = buf[u][f];
      fetch(k + 128 * U, buf[u]);
      if (k < K) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 v = x(r, k);
#pragma unroll
          for (int f = 0; f < FW; ++f) {
            acc[f][r] = fmaf(v.x, now[f].x, acc[f][r]);
            acc[f][r] = fmaf(v.y, now[f].y, acc[f][r]);
            acc[f][r] = fmaf(v.z, now[f].z, acc[f][r]);
            acc[f][r] = fmaf(v.w, now[f].w, acc[f][r]);
          }
        }
      }
    }
  }
}

// Sums of V values over the warp, V a power of two: afterwards lane l holds, in v[0 .. max(1, V / 32) - 1], the totals of the values
// first(l), first(l) + 1, ...; the lanes that differ only in bits below those used hold the same.
template <int V>
__device__ __forceinline__ int qb_sum_values(float (&v)[V], int lane) {
  int first = 0, n = V;
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool upper = lane & stride;
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (i >= n) break;
        const float give = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, stride);
      }
      first += upper ? n : 0;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], stride);
    }
  }
  return first;
}

// Whether lane `lane` is the one that stores what qb_sum_values<V> left (the lowest of the lanes that hold the same).
template <int V>
__device__ __forceinline__ bool qb_sum_stores(int lane) {
  return V >= 32 || (lane & (32 / (V < 32 ? V : 32) - 1)) == 0;
}
