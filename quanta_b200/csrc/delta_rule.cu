// Generalized delta rule with a decay per key channel: a recurrence over time whose state is a matrix
// S [key channel i, value channel j] per (request, head), float32, kept in the request's state slot.
//
//   u   = k / sqrt(sum(k^2) + unit_eps)                       (unit key of the head)
//   w   = exp(-decay_scale * sigmoid(wpre + w_bias))          (decay per key channel)
//   a   = sigmoid(apre + a_bias)                              (removal rate per key channel)
//   S_t = diag(w) S_{t-1} - (a * u) (u^T S_{t-1}) + k v^T     (both terms read the old state)
//   o_t = S_t^T r
//
// A column j of S never meets another column.  Eight lanes share one: lane p has its rows p, p + 8, ..., adds its part of u^T S (and of
// the output) in the order of the rows, and the eight parts meet two by two (lanes 1, 2, 4 apart).  Both kernels below do exactly these
// operations, so a position's numbers depend neither on the cut nor on the batch, not even by rounding.  (Portions once ran in
// chunks of 16 tokens as products, 240 us for the prompt below, whose outputs were 1.7e-7 off float64 against 1.1e-7 here and depended
// on what shared the step.)
//
// The per-head RMS norm with gain and gate that follows is a kernel of the common unit (norm_embed.cu).
#include "common.cuh"

constexpr int DR_LANES = 8;   // lanes that share a column
constexpr int DR_ARRAYS = 5;  // of a (token, head): u, w, a*u, k, r

// What a token does to one row of a column, and to the column's output.
__device__ __forceinline__ float dr_row(float w, float s, float au, float dot, float k, float v) {
  return fmaf(k, v, fmaf(w, s, -(au * dot)));
}
__device__ __forceinline__ float dr_decay(float x, float scale) { return expf(-scale * (1.f / (1.f + expf(-x)))); }
__device__ __forceinline__ float dr_rate(float x) { return 1.f / (1.f + expf(-x)); }
// 1 / |k| of a head, by one warp: the same additions wherever it is called
__device__ __forceinline__ float dr_unit(const float* __restrict__ k, int D, int lane, float unit_eps) {
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) ss = fmaf(k[i], k[i], ss);
  return 1.f / sqrtf(qb_warp_sum(ss) + unit_eps);
}

// ---------------------------------------------------------------------------------------------
// Portions.  A first kernel turns the projections of every (token, head) into the five arrays of [8 RPT] floats in the order in which the
// lanes read them: row i = p + 8 (4 q + e) is number (8 q + p) 4 + e, zeros past D; so lane p's rows are 16-byte pieces, and the
// pieces of the eight lanes lie side by side.  One warp a (token, head).
//
// The recurrence is a chain in time.  A lane group owns one or two columns in registers for the whole portion, a block some columns of one
// (request, head).  Chunks of tokens come into shared memory by asynchronous copies while the chunk before is walked without any barrier.
// One portion alone is bound by the chain of a token (345 cycles: eight multiply-adds, three exchanges, three more, 100 instructions a
// warp): one column a lane, few columns a block.  Enough portions to fill the SMs are bound by the reads of the five arrays from
// shared memory, which two columns a lane halve.  Measured on a B200, token by token with four-byte reads / with this: one portion of
// 2,048 tokens, 32 heads of 64, 618 / 406 us, 8 of 512 615 / 362 (one column a lane 546), 16 heads of 128 962 / 616.
// ---------------------------------------------------------------------------------------------
__global__ void delta_prep_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int a_off,
                                  const float* __restrict__ wpre, const float* __restrict__ a_bias, const float* __restrict__ w_bias,
                                  float* __restrict__ scratch, int T, int H, int D, int DP, float decay_scale, float unit_eps) {
  const int lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= (long)T * H) return;
  const int t = (int)(wid / H), h = (int)(wid % H);
  const float* row = proj + (size_t)t * proj_stride + (size_t)h * D;
  const float inv = dr_unit(row + k_off, D, lane, unit_eps);
  float* to = scratch + (size_t)wid * DR_ARRAYS * DP;
  for (int i = lane; i < DP; i += 32) {
    float u = 0.f, w = 0.f, au = 0.f, k = 0.f, r = 0.f;
    if (i < D) {
      k = row[k_off + i];
      u = k * inv;
      au = dr_rate(row[a_off + i] + a_bias[h * D + i]) * u;
      w = dr_decay(wpre[(size_t)wid * D + i] + w_bias[h * D + i], decay_scale);
      r = row[r_off + i];
    }
    const int p = i & 7, n = i >> 3, at = ((n >> 2) * 8 + p) * 4 + (n & 3);
    to[at] = u; to[DP + at] = w; to[2 * DP + at] = au; to[3 * DP + at] = k; to[4 * DP + at] = r;
  }
}

template <int BYTES>
__device__ __forceinline__ void dr_copy(float* dst_smem, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <int RPT, int C>            // rows of a column a lane holds (D <= DR_LANES * RPT), columns a lane
__global__ void __launch_bounds__(C == 1 ? 128 : 256, 1)
delta_rule_kernel(const float* __restrict__ proj, int proj_stride, int v_off, const float* __restrict__ scratch,
                  float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_start,
                  const int* __restrict__ req_slot, int H, int D, int cols, int chunk) {
  extern __shared__ __align__(16) float sm[];
  constexpr int DP = DR_LANES * RPT, PER = DR_ARRAYS * DP;      // floats of a token's five arrays
  const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int p = tid % DR_LANES, c = tid / DR_LANES * C, col0 = blockIdx.z * cols, j = col0 + c;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (t0 >= t1) return;
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D + j;
  float col[RPT][C];
#pragma unroll
  for (int n = 0; n < RPT; ++n)
#pragma unroll
    for (int e = 0; e < C; ++e) col[n][e] = (j + e < D && p + DR_LANES * n < D) ? S[(size_t)(p + DR_LANES * n) * D + e] : 0.f;
  const int buffer = chunk * (PER + cols);             // [chunk][PER], then v [chunk][cols]
  auto fetch = [&](int c0, int buf) {
    const int n = min(chunk, t1 - c0);
    float* b = sm + (size_t)buf * buffer;
    for (int i = tid; i < n * (PER / 4); i += blockDim.x) {
      const int tt = i / (PER / 4), piece = i % (PER / 4);
      dr_copy<16>(b + 4 * i, scratch + ((size_t)(c0 + tt) * H + h) * PER + 4 * piece);
    }
    for (int i = tid; i < n * cols; i += blockDim.x) {
      const int tt = i / cols, cc = i % cols;
      if (col0 + cc < D) dr_copy<4>(b + chunk * PER + i, proj + (size_t)(c0 + tt) * proj_stride + v_off + (size_t)h * D + col0 + cc);
      else b[chunk * PER + i] = 0.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto rows = [&](const float* from, float (&x)[RPT]) {      // this lane's rows of one array
#pragma unroll
    for (int q = 0; q < RPT / 4; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(from + (q * 8 + p) * 4);
      x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
    }
  };
  auto over_lanes = [&](float (&x)[C], float (&y)[C]) {
#pragma unroll
    for (int o = 1; o < DR_LANES; o <<= 1) {
#pragma unroll
      for (int e = 0; e < C; ++e) x[e] += __shfl_xor_sync(0xffffffffu, x[e], o);
#pragma unroll
      for (int e = 0; e < C; ++e) y[e] += __shfl_xor_sync(0xffffffffu, y[e], o);
    }
  };
  // u of a token and r of the token before meet the same state, so both sums are worked out together
  float u[RPT], r_before[RPT], dot[C], o_before[C];
  auto sums = [&] {
#pragma unroll
    for (int e = 0; e < C; ++e) dot[e] = o_before[e] = 0.f;
#pragma unroll
    for (int n = 0; n < RPT; ++n)
#pragma unroll
      for (int e = 0; e < C; ++e) {
        dot[e] = fmaf(u[n], col[n][e], dot[e]);
        o_before[e] = fmaf(r_before[n], col[n][e], o_before[e]);
      }
    over_lanes(dot, o_before);
  };
  float* to = out + ((size_t)t0 * H + h) * D + j;      // of the token before
  auto store = [&] {
#pragma unroll
    for (int e = 0; e < C; ++e)
      if (p == 0 && j + e < D) to[e] = o_before[e];
    to += (size_t)H * D;
  };
  fetch(t0, 0);
#pragma unroll
  for (int n = 0; n < RPT; ++n) r_before[n] = 0.f;
  bool first = true;
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += chunk, buf ^= 1) {
    const int n_tokens = min(chunk, t1 - c0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                        // this chunk has landed, and everyone is done with the other buffer
    if (c0 + chunk < t1) fetch(c0 + chunk, buf ^ 1);
    const float* at = sm + (size_t)buf * buffer;
    const float* v = at + chunk * PER + c;
    rows(at, u);
    constexpr int UNROLL = C == 1 && RPT <= 16 ? 4 : 1;
#pragma unroll UNROLL
    for (int tt = 0; tt < n_tokens; ++tt, at += PER, v += cols) {
      float w[RPT], au[RPT], k[RPT], vj[C];
      rows(at + DP, w);
      rows(at + 2 * DP, au);
      rows(at + 3 * DP, k);
#pragma unroll
      for (int e = 0; e < C; ++e) vj[e] = v[e];
      sums();
      if (!first) store();
      first = false;
      rows(at + 4 * DP, r_before);
      rows(at + PER, u);                    // behind the last token: whatever lies there, not used
#pragma unroll
      for (int n = 0; n < RPT; ++n)
#pragma unroll
        for (int e = 0; e < C; ++e) col[n][e] = dr_row(w[n], col[n][e], au[n], dot[e], k[n], vj[e]);
    }
  }
  sums();
  store();
#pragma unroll
  for (int n = 0; n < RPT; ++n)
#pragma unroll
    for (int e = 0; e < C; ++e)
      if (j + e < D && p + DR_LANES * n < D) S[(size_t)(p + DR_LANES * n) * D + e] = col[n][e];
}

// ---------------------------------------------------------------------------------------------
// Steps in which every request brings one token: preparation and recurrence in one launch.  A thread takes four columns of its rows, so
// that S is read and written in 16-byte pieces that are asked for before anything else; a warp takes 16 columns, a block 16 to 64 of one
// (request, head).  Bound by the chain of the unit key's sum and two column sums.  8 tokens, 32 heads of 64 (8.4 MB of state): 10.4 us
// as two launches with the columns of S read a float at a time, 4.5 us with this; 64 tokens 51 and 19.
// ---------------------------------------------------------------------------------------------
constexpr int DS_MAX_DIM = 128;

template <int RPT>
__global__ void __launch_bounds__(128)
delta_single_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                    const float* __restrict__ wpre, const float* __restrict__ a_bias, const float* __restrict__ w_bias,
                    float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_start,
                    const int* __restrict__ req_slot, int H, int D, int cols, float decay_scale, float unit_eps) {
  qb_follow();
  constexpr int DP = DR_LANES * RPT;
  __shared__ float s_u[DP], s_w[DP], s_au[DP], s_k[DP], s_r[DP];
  const int tid = threadIdx.x, lane = tid & 31, h = blockIdx.y, r = blockIdx.z;
  const int p = lane >> 2, c = (tid >> 5) * 16 + (lane & 3) * 4, j = blockIdx.x * cols + c;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (t0 >= t1) return;
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D + j;
  const bool owns = c < cols && j < D;      // other warps help with the preparation
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 st[RPT];
#pragma unroll
  for (int n = 0; n < RPT; ++n) {
    const int i = p + DR_LANES * n;
    st[n] = i < D && owns ? *reinterpret_cast<const float4*>(S + (size_t)i * D) : zero;
  }
  auto over_lanes = [&](float4 x) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      x.x += __shfl_xor_sync(0xffffffffu, x.x, o); x.y += __shfl_xor_sync(0xffffffffu, x.y, o);
      x.z += __shfl_xor_sync(0xffffffffu, x.z, o); x.w += __shfl_xor_sync(0xffffffffu, x.w, o);
    }
    return x;
  };
  for (int t = t0; t < t1; ++t) {
    const float* row = proj + (size_t)t * proj_stride + (size_t)h * D;
    float4 v = zero;
    if (owns) v = make_float4(row[v_off + j], row[v_off + j + 1], row[v_off + j + 2], row[v_off + j + 3]);
    for (int i = tid; i < DP; i += blockDim.x) {
      const bool in = i < D;
      s_k[i] = in ? row[k_off + i] : 0.f;
      s_r[i] = in ? row[r_off + i] : 0.f;
      s_w[i] = in ? dr_decay(wpre[((size_t)t * H + h) * D + i] + w_bias[h * D + i], decay_scale) : 0.f;
      s_au[i] = in ? dr_rate(row[a_off + i] + a_bias[h * D + i]) : 0.f;      // the rate; times u below
    }
    const float inv = dr_unit(row + k_off, D, lane, unit_eps);
    for (int i = tid; i < DP; i += blockDim.x) {      // (its own numbers)
      const float u = s_k[i] * inv;
      s_u[i] = u;
      s_au[i] *= u;
    }
    __syncthreads();
    float4 dot = zero;
#pragma unroll
    for (int n = 0; n < RPT; ++n) {
      const float u = s_u[p + DR_LANES * n];
      dot = make_float4(fmaf(u, st[n].x, dot.x), fmaf(u, st[n].y, dot.y), fmaf(u, st[n].z, dot.z), fmaf(u, st[n].w, dot.w));
    }
    dot = over_lanes(dot);
    float4 o = zero;
#pragma unroll
    for (int n = 0; n < RPT; ++n) {
      const int i = p + DR_LANES * n;
      const float w = s_w[i], au = s_au[i], k = s_k[i], rr = s_r[i];
      st[n] = make_float4(dr_row(w, st[n].x, au, dot.x, k, v.x), dr_row(w, st[n].y, au, dot.y, k, v.y),
                          dr_row(w, st[n].z, au, dot.z, k, v.z), dr_row(w, st[n].w, au, dot.w, k, v.w));
      o = make_float4(fmaf(rr, st[n].x, o.x), fmaf(rr, st[n].y, o.y), fmaf(rr, st[n].z, o.z), fmaf(rr, st[n].w, o.w));
    }
    o = over_lanes(o);
    if (p == 0 && owns) *reinterpret_cast<float4*>(out + ((size_t)t * H + h) * D + j) = o;
    if (t + 1 < t1) __syncthreads();
  }
#pragma unroll
  for (int n = 0; n < RPT; ++n) {
    const int i = p + DR_LANES * n;
    if (i < D && owns) *reinterpret_cast<float4*>(S + (size_t)i * D) = st[n];
  }
}

static int dr_rows(int D) { return D <= 32 ? 4 : D <= 64 ? 8 : D <= 128 ? 16 : 32; }

// Floats of scratch that a step wants.
extern "C" long long qb_delta_rule_scratch(int T, int H, int D) {
  return T <= 0 || H <= 0 || D <= 0 || D > 256 ? 0 : (long long)T * H * DR_ARRAYS * DR_LANES * dr_rows(D);
}

// scratch: qb_delta_rule_scratch floats, on 16 bytes
extern "C" int qb_delta_rule(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                             const float* wpre, const float* a_bias, const float* w_bias, float* state,
                             float* out, float* scratch, const int* req_start, const int* req_slot, int R,
                             int T, int H, int D, float decay_scale, float unit_eps, cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  if (D <= 0 || D > 256 || H <= 0) return QB_ERR_UNSUPPORTED;
  const int rpt = dr_rows(D), dp = rpt * DR_LANES;
  if (T == R && D % 4 == 0 && D <= DS_MAX_DIM && H <= 65535 && R <= 65535 && (((uintptr_t)state | (uintptr_t)out) & 15) == 0) {
    // 64 columns a block, or fewer, down to 16, while that leaves SMs without one
    int CB = 64;
    while (CB > 16 && (CB / 2 >= D || (long)R * H * ((D + CB - 1) / CB) < 132)) CB /= 2;
    const dim3 single((D + CB - 1) / CB, H, R);
#define DS_SINGLE(N)                                                                                                             \
  qb_launch(delta_single_kernel<N>, single, 128, 0, stream, proj, proj_stride, r_off, k_off, v_off, a_off, wpre, a_bias, w_bias, \
            state, out, req_start, req_slot, H, D, CB, decay_scale, unit_eps)
    if (rpt == 4) DS_SINGLE(4);
    else if (rpt == 8) DS_SINGLE(8);
    else DS_SINGLE(16);
#undef DS_SINGLE
    QB_LAUNCH_CHECK();
    return 0;
  }
  if (((uintptr_t)scratch & 15) != 0) return QB_ERR_BAD_ARG;
  const long warps = (long)T * H;
  delta_prep_kernel<<<(int)((warps + 3) / 4), 128, 0, stream>>>(proj, proj_stride, r_off, k_off, a_off, wpre, a_bias, w_bias, scratch,
                                                              T, H, D, dp, decay_scale, unit_eps);
  QB_LAUNCH_CHECK();
  // columns a block: all of them (at most 64, or what the registers allow) unless that leaves most SMs idle; then fewer, down to 16
  // where requests bring portions (the block's threads also fetch the chunks) and down to 4 where every request
  // brings one token (the state's bytes are what counts, spread over all SMs); whole warps
  const int min_cols = T > R ? 16 : 4, max_cols = rpt == 32 ? 16 : 64;
  int splits = (D + max_cols - 1) / max_cols;
  while ((long)R * H * splits < 132 && (D + 2 * splits - 1) / (2 * splits) >= min_cols) splits *= 2;
  int cols = (D + splits - 1) / splits;
  const int C = cols > 16 ? 2 : 1;
  cols = (cols + 4 * C - 1) / (4 * C) * (4 * C);
  splits = (D + cols - 1) / cols;
  const int chunk = rpt <= 8 ? 32 : rpt == 16 ? 16 : 8;
  const size_t smem = ((size_t)2 * chunk * (DR_ARRAYS * dp + cols) + DR_ARRAYS * dp) * sizeof(float);      // (reads of u go a token past the end)
  dim3 grid(R, H, splits);
#define DR_LAUNCH(N, C_)                                                                                   \
  do {                                                                                                     \
    auto kern = delta_rule_kernel<N, C_>;                                                                  \
    if (smem > 48 * 1024) {                                                                                \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
      if (e != cudaSuccess) return (int)e;                                                                 \
    }                                                                                                      \
    kern<<<grid, cols / C * DR_LANES, smem, stream>>>(proj, proj_stride, v_off, scratch, state, out, req_start, req_slot, H, D, cols, chunk); \
  } while (0)
  if (rpt == 4 && C == 1) DR_LAUNCH(4, 1);
  else if (rpt == 4) DR_LAUNCH(4, 2);
  else if (rpt == 8 && C == 1) DR_LAUNCH(8, 1);
  else if (rpt == 8) DR_LAUNCH(8, 2);
  else if (rpt == 16 && C == 1) DR_LAUNCH(16, 1);
  else if (rpt == 16) DR_LAUNCH(16, 2);
  else DR_LAUNCH(32, 1);
#undef DR_LAUNCH
  QB_LAUNCH_CHECK();
  return 0;
}

// out[t, c] = tanh(x[t, off + c]) for c < n, in the activation dtype (the inner activation of a
// low-rank pair of projections whose first product sits inside a wider fused product).
template <typename O>
__global__ void tanh_cols_kernel(const float* __restrict__ x, int x_stride, int off, O* __restrict__ out,
                                 int T, int n) {
  qb_follow();
  const size_t total = (size_t)T * n;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t t = i / n, c = i % n;
    out[i] = qb_from_float<O>(tanhf(x[t * x_stride + off + c]));
  }
}

extern "C" int qb_tanh_cols(const float* x, int x_stride, int off, void* out, int out_dtype, int T, int n,
                            cudaStream_t stream) {
  if (T <= 0 || n <= 0) return 0;
  const size_t total = (size_t)T * n;
  const int blocks = (int)((total + 255) / 256 < 2048 ? (total + 255) / 256 : 2048);
  QB_DISPATCH_DTYPE(out_dtype, O, qb_launch(tanh_cols_kernel<O>, blocks, 256, 0, stream, x, x_stride, off, (O*)out, T, n));
  QB_LAUNCH_CHECK();
  return 0;
}
