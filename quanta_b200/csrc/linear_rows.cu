// out[r] = x[r] W^T for a few float32 rows: the projections and the output matrix of a float32 step that decodes.
//
// Bound by the bytes of W.  Measured on a B200 (weights from HBM) beside the library's float32 product of as many rows: 4 rows of
// 2,048 x 3,072 8.4 us against 39 (52 with the spare rows of a bfloat16 step), x 32,000 53 against 79 (4.9 TB/s), 16 rows of 3,072 x 8,192
// 61 against 78; above 16 rows the products of one input no longer fit a warp's registers and the library's tiles win, and above eight of
// more than 8,192 numbers, which are not copied to shared memory (16 rows of 16,384 x 512: 110 us, the library 97).
#include "rows_f32.cuh"

constexpr int LR_WARPS = 4;

struct LinearRows {
  const float *x, *w;
  float* out;
  int rows, K, N;
};

extern __shared__ __align__(16) float lr_smem[];

template <int FW, int U, int R, bool COPIED>
__device__ __forceinline__ void linear_rows_run(const LinearRows& a, int n0, int lane) {
  const float* wr[FW];
#pragma unroll
  for (int f = 0; f < FW; ++f) wr[f] = a.w + (size_t)min(n0 + f, a.N - 1) * a.K;
  float acc[FW][R];
  auto x = [&](int r, int k) {
    const size_t at = (size_t)min(r, a.rows - 1) * a.K + k;
    return COPIED ? *reinterpret_cast<const float4*>(lr_smem + at) : __ldg(reinterpret_cast<const float4*>(a.x + at));
  };
  qb_rows_dot<FW, R, U>(wr, x, [] { if (COPIED) qb_rows_ready(); }, a.K, lane, acc);
  float v[FW * R];                       // index r * FW + f
#pragma unroll
  for (int f = 0; f < FW; ++f)
#pragma unroll
    for (int r = 0; r < R; ++r) v[r * FW + f] = acc[f][r];
  const int first = qb_sum_values<FW * R>(v, lane);
  if (!qb_sum_stores<FW * R>(lane)) return;
  constexpr int HELD = FW * R > 32 ? FW * R / 32 : 1;
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int r = (first + i) / FW, n = n0 + (first + i) % FW;
    if (r < a.rows && n < a.N) a.out[(size_t)r * a.N + n] = v[i];
  }
}

template <int FW, int U, int CAP, bool COPIED>
__global__ void __launch_bounds__(LR_WARPS * 32) linear_rows_kernel(LinearRows a) {
  const int lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * LR_WARPS + (threadIdx.x >> 5)) * FW;       // past N: the last row again, nothing stored
  if (COPIED) qb_rows_copy(lr_smem, [&](int r) { return a.x + (size_t)r * a.K; }, a.rows, a.K);
  if (CAP <= 4 && a.rows <= 1) linear_rows_run<FW, U, 1, COPIED>(a, n0, lane);
  else if (CAP <= 4 && a.rows <= 2) linear_rows_run<FW, U, 2, COPIED>(a, n0, lane);
  else if (CAP <= 4) linear_rows_run<FW, U, 4, COPIED>(a, n0, lane);
  else if (a.rows <= 8) linear_rows_run<FW, U, 8, COPIED>(a, n0, lane);
  else linear_rows_run<FW, U, CAP, COPIED>(a, n0, lane);
}

template <int FW, int U, int CAP>
static int linear_rows_launch(const LinearRows& a, cudaStream_t stream) {
  const int grid = (a.N + FW * LR_WARPS - 1) / (FW * LR_WARPS), smem = qb_rows_smem(a.rows, a.K);
  if (smem > 0) {
    const cudaError_t err = cudaFuncSetAttribute(linear_rows_kernel<FW, U, CAP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 QB_ROWS_SMEM);
    if (err != cudaSuccess) return (int)err;
    linear_rows_kernel<FW, U, CAP, true><<<grid, LR_WARPS * 32, smem, stream>>>(a);
  } else {
    linear_rows_kernel<FW, U, CAP, false><<<grid, LR_WARPS * 32, 0, stream>>>(a);
  }
  QB_LAUNCH_CHECK();
  return 0;
}

// rows <= 16; K a multiple of 4; x and w on 16 bytes.
extern "C" int qb_linear_rows(const float* x, const float* w, float* out, int rows, int K, int N, cudaStream_t stream) {
  if (rows <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 4 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return QB_ERR_BAD_ARG;
  if (rows > 16) return QB_ERR_UNSUPPORTED;
  const LinearRows a{x, w, out, rows, K, N};
  // up to four rows: two rows of weights a warp, four steps ahead (more warps for narrow matrices); above, four rows of weights a
  // warp, so that an input row read serves four products
  return rows <= 4 ? linear_rows_launch<2, 4, 4>(a, stream) : linear_rows_launch<4, 2, 16>(a, stream);
}
