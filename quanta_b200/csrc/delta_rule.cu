// Generalized delta rule with a decay per key channel: a recurrence over time whose state is a matrix
// S [key channel i, value channel j] per (request, head), float32, kept in the request's state slot.
//
//   u   = k / sqrt(sum(k^2) + unit_eps)                       (unit key of the head)
//   w   = exp(-decay_scale * sigmoid(wpre + w_bias))          (decay per key channel)
//   a   = sigmoid(apre + a_bias)                              (removal rate per key channel)
//   S_t = diag(w) S_{t-1} - (a * u) (u^T S_{t-1}) + k v^T     (both terms read the old state)
//   o_t = S_t^T r
//
// A first kernel turns the projections of every (token, head) into w, a*u and u (all tokens at once).  The
// recurrence itself is a chain in time.
//
// Two forms.  Token by token (decoding, short portions, large heads): a column j of S never meets another column, so eight neighbouring
// lanes own one column (rows i = p, p + 8, ... for lane p) in registers for the whole step, and a block owns
// some columns of one (request, head).  Tokens are taken in chunks: w, a*u, u, k, r, v of the next chunk come
// into shared memory by asynchronous copies while every lane group walks the chunk before without any
// barrier.
//
// Chunks of 16 tokens (portions of prompts): inside a chunk the recurrence is unrolled into products, see below.  Between the two
// forms a position's numbers differ by float32 rounding.
//
// The per-head RMS norm with gain and gate that follows is a kernel of the common unit (norm_embed.cu).
#include "common.cuh"

constexpr int DR_LANES = 8;   // lanes that share a column
constexpr int DR_MAX_COLS = 64;    // columns a block (512 threads), so that a lane's rows stay in registers
template <int RPT> struct DrThreads { static constexpr int max = RPT * 64 < 512 ? RPT * 64 : 512; };

// w, a*u and u of every (token, head), float32 [T, H, D] each: one warp a (token, head), the sum over k^2 a
// warp reduction in a fixed order.
__global__ void delta_prep_kernel(const float* __restrict__ proj, int proj_stride, int k_off, int a_off,
                                  const float* __restrict__ wpre, const float* __restrict__ a_bias,
                                  const float* __restrict__ w_bias, float* __restrict__ w_out,
                                  float* __restrict__ au_out, float* __restrict__ u_out, int T, int H, int D,
                                  float decay_scale, float unit_eps) {
  const int lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= (long)T * H) return;
  const int t = (int)(wid / H), h = (int)(wid % H);
  const float* row = proj + (size_t)t * proj_stride + (size_t)h * D;
  const size_t base = ((size_t)t * H + h) * D;
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) { const float kv = row[k_off + i]; ss += kv * kv; }
  ss = qb_warp_sum(ss);
  const float inv = 1.f / sqrtf(ss + unit_eps);
  for (int i = lane; i < D; i += 32) {
    const float uv = row[k_off + i] * inv;
    const float av = 1.f / (1.f + expf(-(row[a_off + i] + a_bias[h * D + i])));
    const float sg = 1.f / (1.f + expf(-(wpre[base + i] + w_bias[h * D + i])));
    w_out[base + i] = expf(-decay_scale * sg);
    au_out[base + i] = av * uv;
    u_out[base + i] = uv;
  }
}

__device__ __forceinline__ void dr_copy4(float* dst_smem, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <int RPT>            // rows of the column a lane holds: D <= DR_LANES * RPT
__global__ void __launch_bounds__(DrThreads<RPT>::max, 1)
delta_rule_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off,
                  const float* __restrict__ w_in, const float* __restrict__ au_in, const float* __restrict__ u_in,
                  float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_start,
                  const int* __restrict__ req_slot, int H, int D, int cols_per_block, int chunk) {
  extern __shared__ float sm[];
  constexpr int DP = DR_LANES * RPT;       // padded key channels (a power of two)
  const int r = blockIdx.x, h = blockIdx.y;
  const int col0 = blockIdx.z * cols_per_block;
  const int tid = threadIdx.x;
  const int p = tid % DR_LANES;
  const int j = col0 + tid / DR_LANES;
  const bool owns = (tid / DR_LANES) < cols_per_block && j < D;
  const size_t plane = (size_t)chunk * DP;  // one array of a chunk; six arrays a buffer, two buffers
  // the padding rows (i >= D) are read as zeros and never written
  for (size_t i = tid; i < 12 * plane; i += blockDim.x) sm[i] = 0.f;

  const int t0 = req_start[r], t1 = req_start[r + 1];
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D;
  float col[RPT];
#pragma unroll
  for (int ii = 0; ii < RPT; ++ii) {
    const int i = p + DR_LANES * ii;
    col[ii] = (owns && i < D) ? S[(size_t)i * D + j] : 0.f;
  }
  __syncthreads();

  // a chunk's six arrays come in by asynchronous copies while the chunk before is walked
  auto fetch = [&](int c0, int buf) {
    const int n = min(chunk, t1 - c0);
    float* b = sm + (size_t)buf * 6 * plane;
    for (int idx = tid; idx < n * DP; idx += blockDim.x) {
      const int tt = idx / DP, i = idx % DP;
      if (i < D) {
        const size_t g = ((size_t)(c0 + tt) * H + h) * D + i;
        const float* row = proj + (size_t)(c0 + tt) * proj_stride + (size_t)h * D + i;
        dr_copy4(b + idx, w_in + g);
        dr_copy4(b + plane + idx, au_in + g);
        dr_copy4(b + 2 * plane + idx, u_in + g);
        dr_copy4(b + 3 * plane + idx, row + k_off);
        dr_copy4(b + 4 * plane + idx, row + r_off);
        dr_copy4(b + 5 * plane + idx, row + v_off);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (t0 < t1) fetch(t0, 0);
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += chunk, buf ^= 1) {
    const int n = min(chunk, t1 - c0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                        // this chunk has landed, and everyone is done with the other buffer
    if (c0 + chunk < t1) fetch(c0 + chunk, buf ^ 1);
    const float* s_w = sm + (size_t)buf * 6 * plane;
    const float* s_au = s_w + plane;
    const float* s_u = s_au + plane;
    const float* s_k = s_u + plane;
    const float* s_r = s_k + plane;
    const float* s_v = s_r + plane;
    for (int tt = 0; tt < n; ++tt) {
      const size_t o = (size_t)tt * DP;
      float dot = 0.f;
#pragma unroll
      for (int ii = 0; ii < RPT; ++ii) dot += s_u[o + p + DR_LANES * ii] * col[ii];
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      dot += __shfl_xor_sync(0xffffffffu, dot, 4);
      const float vj = owns ? s_v[o + j] : 0.f;
      float acc = 0.f;
#pragma unroll
      for (int ii = 0; ii < RPT; ++ii) {
        const int i = p + DR_LANES * ii;
        const float s_new = s_w[o + i] * col[ii] - s_au[o + i] * dot + s_k[o + i] * vj;
        col[ii] = s_new;
        acc += s_r[o + i] * s_new;
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      if (owns && p == 0) out[((size_t)(c0 + tt) * H + h) * D + j] = acc;
    }
  }
#pragma unroll
  for (int ii = 0; ii < RPT; ++ii) {
    const int i = p + DR_LANES * ii;
    if (owns && i < D) S[(size_t)i * D + j] = col[ii];
  }
}

// ---------------------------------------------------------------------------------------------
// Steps in which every request brings one token: preparation and recurrence in one launch.  A block takes CB columns of one (request,
// head) with 256 threads: c4 = CB / 4 groups of four columns x 256 / c4 groups of rows, so that S is read and written in 16-byte pieces
// that are asked for before anything else; the sums over the rows go over the lanes and then over the eight warps.  Bound by its
// chain of two block sums.  8 tokens, 32 heads of 64 (8.4 MB of state): 10.4 us as two launches with the columns of S read a float at a
// time, 4.5 us with this; one token 8.4 and 3.7.
// ---------------------------------------------------------------------------------------------
constexpr int DS_THREADS = 256, DS_MAX_DIM = 128;

template <int NR>                                   // rows a thread
__global__ void __launch_bounds__(DS_THREADS)
delta_single_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                    const float* __restrict__ wpre, const float* __restrict__ a_bias, const float* __restrict__ w_bias,
                    float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_start,
                    const int* __restrict__ req_slot, int H, int D, int c4, float decay_scale, float unit_eps) {
  qb_follow();
  __shared__ float s_u[DS_MAX_DIM], s_w[DS_MAX_DIM], s_au[DS_MAX_DIM], s_k[DS_MAX_DIM], s_r[DS_MAX_DIM], s_ss[8];
  __shared__ __align__(16) float4 s_dot[8][16], s_out[8][16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, r = blockIdx.z;
  const int c = tid % c4, rg = tid / c4, RG = DS_THREADS / c4, j = (blockIdx.x * c4 + c) * 4;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (t0 >= t1) return;
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D + j;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 st[NR];
#pragma unroll
  for (int n = 0; n < NR; ++n) {
    const int i = rg + RG * n;
    st[n] = i < D && j < D ? *reinterpret_cast<const float4*>(S + (size_t)i * D) : zero;
  }
  auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
  // the sum over a block's rows of four columns: over the lanes of a column, then over the warps in order
  auto over_rows = [&](float4 p, float4 (&buf)[8][16]) {
    for (int o = c4; o < 32; o <<= 1)
      p = add(p, make_float4(__shfl_xor_sync(0xffffffffu, p.x, o), __shfl_xor_sync(0xffffffffu, p.y, o),
                             __shfl_xor_sync(0xffffffffu, p.z, o), __shfl_xor_sync(0xffffffffu, p.w, o)));
    if (lane < c4) buf[warp][c] = p;
    __syncthreads();
    float4 sum = buf[0][c];
#pragma unroll
    for (int w = 1; w < 8; ++w) sum = add(sum, buf[w][c]);
    return sum;
  };
  for (int t = t0; t < t1; ++t) {
    const float* row = proj + (size_t)t * proj_stride + (size_t)h * D;
    float4 v = zero;
    if (j < D) v = make_float4(row[v_off + j], row[v_off + j + 1], row[v_off + j + 2], row[v_off + j + 3]);
    float kv = 0.f, w = 1.f, a = 0.f;
    if (tid < D) {
      kv = row[k_off + tid];
      a = 1.f / (1.f + expf(-(row[a_off + tid] + a_bias[h * D + tid])));
      w = expf(-decay_scale * (1.f / (1.f + expf(-(wpre[((size_t)t * H + h) * D + tid] + w_bias[h * D + tid])))));
      s_r[tid] = row[r_off + tid];
      s_k[tid] = kv;
      s_w[tid] = w;
    }
    const float part = qb_warp_sum(kv * kv);        // warps past D add zeros
    if (lane == 0) s_ss[warp] = part;
    __syncthreads();
    float ss = s_ss[0];
#pragma unroll
    for (int q = 1; q < DS_MAX_DIM / 32; ++q) ss += s_ss[q];
    if (tid < D) {
      const float u = kv * (1.f / sqrtf(ss + unit_eps));
      s_u[tid] = u;
      s_au[tid] = a * u;
    }
    __syncthreads();
    float4 p = zero;
#pragma unroll
    for (int n = 0; n < NR; ++n) {
      const int i = rg + RG * n;
      const float u = i < D ? s_u[i] : 0.f;
      p = make_float4(fmaf(u, st[n].x, p.x), fmaf(u, st[n].y, p.y), fmaf(u, st[n].z, p.z), fmaf(u, st[n].w, p.w));
    }
    const float4 dot = over_rows(p, s_dot);
    p = zero;
#pragma unroll
    for (int n = 0; n < NR; ++n) {
      const int i = rg + RG * n;
      if (i < D) {
        const float wi = s_w[i], ai = s_au[i], ki = s_k[i], ri = s_r[i];
        st[n] = make_float4(wi * st[n].x - ai * dot.x + ki * v.x, wi * st[n].y - ai * dot.y + ki * v.y,
                            wi * st[n].z - ai * dot.z + ki * v.z, wi * st[n].w - ai * dot.w + ki * v.w);
        p = make_float4(fmaf(ri, st[n].x, p.x), fmaf(ri, st[n].y, p.y), fmaf(ri, st[n].z, p.z), fmaf(ri, st[n].w, p.w));
      }
    }
    const float4 o = over_rows(p, s_out);
    if (rg == 0 && j < D) *reinterpret_cast<float4*>(out + ((size_t)t * H + h) * D + j) = o;
    if (t + 1 < t1) __syncthreads();
  }
#pragma unroll
  for (int n = 0; n < NR; ++n) {
    const int i = rg + RG * n;
    if (i < D && j < D) *reinterpret_cast<float4*>(S + (size_t)i * D) = st[n];
  }
}

// ---------------------------------------------------------------------------------------------
// Chunks of DC = 16 tokens, all in float32.  With W_t the product of the decays of the chunk's tokens up to t, z = -a u and
// y_t = S_{t-1}^T u_t, the recurrence from the state S at the chunk's start is
//     S_t = W_t S + sum_{s <= t} (W_t / W_s) (z_s y_s^T + k_s v_s^T),
// so that y, the outputs and the state at the chunk's end are linear in S and v, with coefficients that do not depend on S:
//     y = U S (+ G v),   o = R S + N v,   S' = W S + Z^T (U S) + K^T v.
// `delta_chunk_kernel` works U, R, Z, K [16, D], N [16, 16] and W [D] out for every (chunk, head) at once: the 16 x 16 products of
// u W, r W with z / W, k / W, a unit triangular system solved column by column, two more triangular products.  (Dividing by W costs
// one rounding: with the launch rule below W is above 1e-17.)  `delta_states_kernel` then walks the chunks, a block 16 columns of
// one (request, head): 48 x D x 16 FMAs three times a chunk instead of 16 dependent steps.  Sums over s run over tokens up to t only,
// so a token's infinities reach no earlier token.  Padding tokens of the last chunk have w = 1 and zeros elsewhere.
//
// Measured on a B200, one prompt of 2,048 tokens, 32 heads of 64: 595 us token by token; 72 + 178 us (the walk reads and writes shared
// memory in 70 to 80 % of the cycles).  Against float64 the outputs are 1.7e-7 off in the 2-norm (token by token 1.1e-7), the state
// 1.0e-7 (0.8e-7).
// ---------------------------------------------------------------------------------------------
constexpr int DC = 16, DC_COLS = 16, DC_THREADS = 128, DC_WALKERS = 256;

template <int DP> struct DcLayout {                 // floats of one (chunk, head)
  static constexpr int U = 0, R = DC * DP, Z = 2 * DC * DP, K = 3 * DC * DP, N = 4 * DC * DP, W = N + DC * DC, SIZE = W + DP;
};

// Chunk `c` of all requests' chunks: its first token and the end of its request; false if there are fewer.  One warp.
__device__ __forceinline__ bool dc_find(const int* __restrict__ req_start, int R, int c, int lane, int& first, int& end) {
  int before = 0;
  for (int r0 = 0; r0 < R; r0 += 32) {
    const int r = r0 + lane;
    const int a = r < R ? req_start[r] : 0, b = r < R ? req_start[r + 1] : 0, n = (b - a + DC - 1) / DC;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, c < before + sum);
    if (hit) {
      const int l = __ffs(hit) - 1;
      first = __shfl_sync(0xffffffffu, a + (c - before - sum + n) * DC, l);
      end = __shfl_sync(0xffffffffu, b, l);
      return true;
    }
    before += __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}

// Chunks of the requests before `upto`.  One warp.
__device__ __forceinline__ int dc_before(const int* __restrict__ req_start, int upto, int lane) {
  int n = 0;
  for (int r = lane; r < upto; r += 32) n += (req_start[r + 1] - req_start[r] + DC - 1) / DC;
  return (int)__reduce_add_sync(0xffffffffu, (unsigned)n);
}

template <int DP>
__global__ void __launch_bounds__(DP + 64 > DC_THREADS ? DP + 64 : DC_THREADS)
delta_chunk_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int a_off, const float* __restrict__ wpre,
                   const float* __restrict__ a_bias, const float* __restrict__ w_bias, float* __restrict__ coef,
                   const int* __restrict__ req_start, int R, int H, int D, float decay_scale, float unit_eps) {
  using L = DcLayout<DP>;
  constexpr int LD = DP + 4, PER = DP / 32;
  __shared__ __align__(16) float s_u[DC][LD], s_r[DC][LD], s_z[DC][LD], s_k[DC][LD], s_w[DC][DP];
  __shared__ __align__(16) float s_L[DC][DC], s_M[DC][DC], s_P[DC][DC], s_Q[DC][DC];      // [t][s]
  __shared__ int s_first, s_end;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y;
  if (warp == 0) {
    int first = 0, end = 0;
    const bool found = dc_find(req_start, R, blockIdx.x, lane, first, end);
    if (lane == 0) { s_first = first; s_end = found ? end : first; }
  }
  __syncthreads();
  const int t0 = s_first, n = min(DC, s_end - t0);
  if (n <= 0) return;                               // the grid is the most chunks there can be
  // the tokens' u, r, z, k, w: a warp four tokens, everything they read asked for at once
  if (warp < DC / 4) {
    float kv[4][PER], rv[4][PER], av[4][PER], wv[4][PER], ab[PER], wb[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int i = lane + 32 * q;
      ab[q] = i < D ? a_bias[h * D + i] : 0.f;
      wb[q] = i < D ? w_bias[h * D + i] : 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = warp * 4 + e;
        const bool in = t < n && i < D;
        const float* row = proj + (size_t)(t0 + (in ? t : 0)) * proj_stride + (size_t)h * D + (in ? i : 0);
        kv[e][q] = in ? row[k_off] : 0.f;
        rv[e][q] = in ? row[r_off] : 0.f;
        av[e][q] = in ? row[a_off] : 0.f;
        wv[e][q] = in ? wpre[((size_t)(t0 + t) * H + h) * D + i] : 0.f;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = warp * 4 + e;
      float ss = 0.f;
#pragma unroll
      for (int q = 0; q < PER; ++q) ss += kv[e][q] * kv[e][q];
      ss = qb_warp_sum(ss);
      const float inv = 1.f / sqrtf(ss + unit_eps);
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int i = lane + 32 * q;
        const bool in = t < n && i < D;
        const float uv = in ? kv[e][q] * inv : 0.f;
        const float a = 1.f / (1.f + expf(-(av[e][q] + ab[q])));
        const float sg = 1.f / (1.f + expf(-(wv[e][q] + wb[q])));
        s_u[t][i] = uv;
        s_r[t][i] = rv[e][q];
        s_z[t][i] = in ? -(a * uv) : 0.f;
        s_k[t][i] = kv[e][q];
        s_w[t][i] = in ? expf(-decay_scale * sg) : 1.f;
      }
    }
  }
  __syncthreads();
  float w_end = 1.f;
  if (tid < DP) {                                   // u W_{t-1}, r W_t, z / W_t, k / W_t
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      s_u[t][tid] *= w_end;
      w_end *= s_w[t][tid];
      const float inv = 1.f / w_end;
      s_r[t][tid] *= w_end;
      s_z[t][tid] *= inv;
      s_k[t][tid] *= inv;
    }
  }
  __syncthreads();
  // 32 x 32 products over the channels: rows u, r; columns z, k; a thread 4 x 2 of them
  if (tid < DC_THREADS) {
    const int rg = tid >> 4, cg = tid & 15;
    float acc[4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = 0.f;
#pragma unroll 4
    for (int i = 0; i < DP; i += 4) {
      const float4 x[4] = {*reinterpret_cast<const float4*>(&s_u[rg][i]), *reinterpret_cast<const float4*>(&s_u[rg + 8][i]),
                           *reinterpret_cast<const float4*>(&s_r[rg][i]), *reinterpret_cast<const float4*>(&s_r[rg + 8][i])};
      const float4 y[2] = {*reinterpret_cast<const float4*>(&s_z[cg][i]), *reinterpret_cast<const float4*>(&s_k[cg][i])};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          acc[a][b] = fmaf(x[a].x, y[b].x, acc[a][b]);
          acc[a][b] = fmaf(x[a].y, y[b].y, acc[a][b]);
          acc[a][b] = fmaf(x[a].z, y[b].z, acc[a][b]);
          acc[a][b] = fmaf(x[a].w, y[b].w, acc[a][b]);
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int t = rg + 8 * a;
      s_L[t][cg] = acc[a][0];
      s_M[t][cg] = acc[a][1];
      s_P[t][cg] = acc[2 + a][0];
      s_Q[t][cg] = acc[2 + a][1];
    }
  }
  __syncthreads();
  float* c = coef + ((size_t)blockIdx.x * H + h) * L::SIZE;
  float y[DC];
  if (tid < DP) {                                   // a channel's column of U, then of R
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float v = s_u[t][tid];
#pragma unroll
      for (int s = 0; s < t; ++s) v = fmaf(s_L[t][s], y[s], v);
      y[t] = v;
      c[L::U + t * DP + tid] = v;
    }
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float v = s_r[t][tid];
#pragma unroll
      for (int s = 0; s <= t; ++s) v = fmaf(s_P[t][s], y[s], v);
      c[L::R + t * DP + tid] = v;
      c[L::Z + t * DP + tid] = w_end * s_z[t][tid];
    }
    c[L::W + tid] = w_end;
  } else if (tid < DP + DC) {                       // a token's column of G (kept in place of M), then of N
    const int j = tid - DP;
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float v = t > j ? s_M[t][j] : 0.f;
#pragma unroll
      for (int s = 0; s < t; ++s)
        if (s > j) v = fmaf(s_L[t][s], y[s], v);
      y[t] = v;
      s_M[t][j] = v;
    }
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float v = t >= j ? s_Q[t][j] : 0.f;
#pragma unroll
      for (int s = 0; s <= t; ++s)
        if (s > j) v = fmaf(s_P[t][s], y[s], v);
      c[L::N + t * DC + j] = v;
    }
  }
  __syncthreads();
  if (tid < DP) {
#pragma unroll
    for (int s = 0; s < DC; ++s) {
      float v = s_k[s][tid];
#pragma unroll
      for (int t = s + 1; t < DC; ++t) v = fmaf(s_M[t][s], s_z[t][tid], v);
      c[L::K + s * DP + tid] = w_end * v;
    }
  }
}

__device__ __forceinline__ void dc_copy16(float* dst_smem, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

template <int DP> struct DcShared {
  static constexpr int LD = DP + 4, VLD = DC_COLS + 4;
  float a[2][4 * DC][LD];                           // rows U, R, Z, K of a chunk
  float nw[2][DC * DC + DP];                        // N, W
  float v[2][DC][VLD];
  float y[DC][VLD];                                 // U S
  float st[DC_COLS][LD];                            // the state, a column after the other
  union {
    float p1[4][DC][VLD];                           // parts of U S, a warp each
    float p2[4][DC_COLS][LD];                       // parts of Z^T y + K^T v
  };
  float po[4][DC][VLD];                             // parts of R S
};

template <int DP>
__global__ void __launch_bounds__(DC_WALKERS)
delta_states_kernel(const float* __restrict__ proj, int proj_stride, int v_off, const float* __restrict__ coef,
                    float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_start,
                    const int* __restrict__ req_slot, int H, int D) {
  using L = DcLayout<DP>;
  using Sh = DcShared<DP>;
  extern __shared__ __align__(16) unsigned char dc_raw[];
  Sh& sh = *reinterpret_cast<Sh*>(dc_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 3;
  const bool outputs = tid >= DC_THREADS;           // warps 0 .. 3 carry the state on, warps 4 .. 7 work the outputs out beside them
  // the last request's blocks come first: a step's single tokens stand before the portions of prompts
  const int r = gridDim.z - 1 - blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * DC_COLS;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (t0 >= t1) return;
  const bool whole = D % 4 == 0 && ((uintptr_t)out & 15) == 0;      // outputs go out in 16-byte pieces
  const int chunk0 = dc_before(req_start, r, lane);
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D;
  for (int i = tid; i < DC_COLS * DP; i += DC_WALKERS) {
    const int j = i % DC_COLS, ch = i / DC_COLS;
    sh.st[j][ch] = ch < D && col0 + j < D ? S[(size_t)ch * D + col0 + j] : 0.f;
  }
  auto fetch = [&](int c, int b) {
    const float* from = coef + ((size_t)(chunk0 + c) * H + h) * L::SIZE;
    for (int i = tid; i < 4 * DC * DP / 4; i += DC_WALKERS) dc_copy16(&sh.a[b][i / (DP / 4)][i % (DP / 4) * 4], from + 4 * i);
    for (int i = tid; i < (DC * DC + DP) / 4; i += DC_WALKERS) dc_copy16(&sh.nw[b][4 * i], from + L::N + 4 * i);
    for (int i = tid; i < DC * DC_COLS; i += DC_WALKERS) {
      const int t = i / DC_COLS, j = i % DC_COLS, tok = t0 + c * DC + t;
      if (tok < t1 && col0 + j < D) dr_copy4(&sh.v[b][t][j], proj + (size_t)tok * proj_stride + v_off + (size_t)h * D + col0 + j);
      else sh.v[b][t][j] = 0.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int chunks = (t1 - t0 + DC - 1) / DC;
  fetch(0, 0);
  // first product (16 rows x 16 columns over the channels): lanes 2 (halves of a warp's channels) x 4 (rows mg + 4 r) x 4 (columns
  // jg + 4 c)
  const int half = lane >> 4, mg = (lane >> 2) & 3, jg = lane & 3;
  // second product: lanes 8 (channels 4 ig + 32 e) x 4 (columns 4 jg ..)
  const int ig = lane >> 2;
  for (int c = 0; c < chunks; ++c) {
    const int b = c & 1;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                // the chunk has landed, the state is written, the other buffer is free
    if (c + 1 < chunks) fetch(c + 1, b ^ 1);
    {
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
      constexpr int PART = DP / 8;                  // channels of half a warp
      const int row0 = outputs ? DC : 0;            // rows U, or rows R
#pragma unroll
      for (int k = 0; k < PART; k += 4) {
        const int ch = (warp * 2 + half) * PART + k;
        float4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(&sh.a[b][row0 + mg + 4 * i][ch]);
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(&sh.st[jg + 4 * j][ch]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j] = fmaf(x[i].x, y[j].x, acc[i][j]);
            acc[i][j] = fmaf(x[i].y, y[j].y, acc[i][j]);
            acc[i][j] = fmaf(x[i].z, y[j].z, acc[i][j]);
            acc[i][j] = fmaf(x[i].w, y[j].w, acc[i][j]);
          }
      }
      // the halves add: each keeps two of the rows
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float give = half ? acc[i][j] : acc[i + 2][j], keep = half ? acc[i + 2][j] : acc[i][j];
          const float sum = keep + __shfl_xor_sync(0xffffffffu, give, 16);
          (outputs ? sh.po : sh.p1)[warp][mg + 4 * (i + 2 * half)][jg + 4 * j] = sum;
        }
    }
    __syncthreads();
    if (!outputs) {
      const int m = tid >> 3, j = (tid & 7) * 2;
      float2 v = *reinterpret_cast<const float2*>(&sh.p1[0][m][j]);
#pragma unroll
      for (int w = 1; w < 4; ++w) {
        const float2 p = *reinterpret_cast<const float2*>(&sh.p1[w][m][j]);
        v = make_float2(v.x + p.x, v.y + p.y);
      }
      *reinterpret_cast<float2*>(&sh.y[m][j]) = v;
      asm volatile("bar.sync 1, 128;" ::: "memory");          // the four state warps
      // tokens 4 w .. 4 w + 3 of y and of v for warp w
      float4 acc[DP / 32][4];
#pragma unroll
      for (int e = 0; e < DP / 32; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[e][q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int t = warp * 4 + (q & 3);
        const float4 x = *reinterpret_cast<const float4*>(q < 4 ? &sh.y[t][jg * 4] : &sh.v[b][t][jg * 4]);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < DP / 32; ++e) {
          const float4 a = *reinterpret_cast<const float4*>(&sh.a[b][(q < 4 ? 2 : 3) * DC + t][ig * 4 + 32 * e]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            acc[e][i].x = fmaf(a.x, xs[i], acc[e][i].x);
            acc[e][i].y = fmaf(a.y, xs[i], acc[e][i].y);
            acc[e][i].z = fmaf(a.z, xs[i], acc[e][i].z);
            acc[e][i].w = fmaf(a.w, xs[i], acc[e][i].w);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < DP / 32; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) *reinterpret_cast<float4*>(&sh.p2[warp][jg * 4 + q][ig * 4 + 32 * e]) = acc[e][q];
    } else {
      const int t = (tid - DC_THREADS) >> 3, j = (tid & 7) * 2, tok = t0 + c * DC + t;
      float2 v = *reinterpret_cast<const float2*>(&sh.po[0][t][j]);
#pragma unroll
      for (int w = 1; w < 4; ++w) {
        const float2 p = *reinterpret_cast<const float2*>(&sh.po[w][t][j]);
        v = make_float2(v.x + p.x, v.y + p.y);
      }
#pragma unroll
      for (int s = 0; s < DC; ++s) {
        if (s <= t) {
          const float f = sh.nw[b][t * DC + s];
          const float2 x = *reinterpret_cast<const float2*>(&sh.v[b][s][j]);
          v = make_float2(fmaf(f, x.x, v.x), fmaf(f, x.y, v.y));
        }
      }
      if (tok < t1) {
        float* o = out + ((size_t)tok * H + h) * D + col0 + j;
        if (whole) {
          if (col0 + j < D) *reinterpret_cast<float2*>(o) = v;
        } else {
          if (col0 + j < D) o[0] = v.x;
          if (col0 + j + 1 < D) o[1] = v.y;
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < DC_COLS * DP / 4; i += DC_WALKERS) {
      const int j = i / (DP / 4), ch = i % (DP / 4) * 4;
      float4* st = reinterpret_cast<float4*>(&sh.st[j][ch]);
      const float4 w = *reinterpret_cast<const float4*>(&sh.nw[b][DC * DC + ch]);
      float4 v = *st;
      v = make_float4(w.x * v.x, w.y * v.y, w.z * v.z, w.w * v.w);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 p = *reinterpret_cast<const float4*>(&sh.p2[q][j][ch]);
        v = make_float4(v.x + p.x, v.y + p.y, v.z + p.z, v.w + p.w);
      }
      *st = v;
    }
  }
  __syncthreads();
  for (int i = tid; i < DC_COLS * DP; i += DC_WALKERS) {
    const int j = i % DC_COLS, ch = i / DC_COLS;
    if (ch < D && col0 + j < D) S[(size_t)ch * D + col0 + j] = sh.st[j][ch];
  }
}

template <int DP>
static int delta_by_chunks(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off, const float* wpre,
                           const float* a_bias, const float* w_bias, float* state, float* out, float* coef, const int* req_start,
                           const int* req_slot, int R, int T, int H, int D, float decay_scale, float unit_eps, cudaStream_t stream) {
  constexpr int threads = DP + 64 > DC_THREADS ? DP + 64 : DC_THREADS;
  delta_chunk_kernel<DP><<<dim3(T / DC + R, H), threads, 0, stream>>>(proj, proj_stride, r_off, k_off, a_off, wpre, a_bias, w_bias,
                                                                      coef, req_start, R, H, D, decay_scale, unit_eps);
  QB_LAUNCH_CHECK();
  static const cudaError_t once = cudaFuncSetAttribute(delta_states_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)sizeof(DcShared<DP>));
  if (once != cudaSuccess) return (int)once;
  delta_states_kernel<DP><<<dim3((D + DC_COLS - 1) / DC_COLS, H, R), DC_WALKERS, sizeof(DcShared<DP>), stream>>>(
      proj, proj_stride, v_off, coef, state, out, req_start, req_slot, H, D);
  QB_LAUNCH_CHECK();
  return 0;
}

// Whether a step runs in chunks.  `longest`: tokens of the longest portion.  Token by token a launch takes as long as its longest
// portion (0.29 us a token), in chunks 0.11 us a token and 4 us more for two launches, and every request, of one token too, costs its blocks a
// chunk.  Measured at 32 heads of 64, token by token and in chunks: one portion of 32 tokens 15.5 and 14.5 us, 128 42 and 23, 2,048 595 and 240;
// 8 of 20 30 and 38, 8 of 64 77 and 61; 24 single tokens with one portion of 200 122 and 78, of 512 277 and 107; 16 heads of 128, one of
// 2,048: 941 and 361.  decay_scale bounds the chunk's product of decays: above e^-40.
static bool delta_in_chunks(int R, int H, int D, int longest, float decay_scale) {
  return D <= 128 && H <= 65535 && R <= 65535 && longest >= 32 && longest >= 6 * R && decay_scale >= 0.f && decay_scale * DC <= 40.f;
}
static int delta_padded(int D) { return D <= 32 ? 32 : D <= 64 ? 64 : 128; }

// Floats of scratch that a step wants.
extern "C" long long qb_delta_rule_scratch(int R, int T, int H, int D, int longest, float decay_scale) {
  if (R <= 0 || T <= 0 || H <= 0 || D <= 0) return 0;
  if (!delta_in_chunks(R, H, D, longest, decay_scale)) return 3LL * T * H * D;
  const int DP = delta_padded(D);
  return (long long)(T / DC + R) * H * (4 * DC * DP + DC * DC + DP);
}

// scratch: qb_delta_rule_scratch floats, on 16 bytes
extern "C" int qb_delta_rule(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                             const float* wpre, const float* a_bias, const float* w_bias, float* state,
                             float* out, float* scratch, const int* req_start, const int* req_slot, int R,
                             int T, int H, int D, int longest, float decay_scale, float unit_eps, cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  if (D <= 0 || D > 256 || H <= 0) return QB_ERR_UNSUPPORTED;
  if (delta_in_chunks(R, H, D, longest, decay_scale)) {
#define DC_ARGS proj, proj_stride, r_off, k_off, v_off, a_off, wpre, a_bias, w_bias, state, out, scratch, req_start, req_slot, R, T, H, \
                D, decay_scale, unit_eps, stream
    switch (delta_padded(D)) {
      case 32: return delta_by_chunks<32>(DC_ARGS);
      case 64: return delta_by_chunks<64>(DC_ARGS);
      default: return delta_by_chunks<128>(DC_ARGS);
    }
#undef DC_ARGS
  }
  if (T == R && D % 4 == 0 && D <= DS_MAX_DIM && H <= 65535 && R <= 65535 && (((uintptr_t)state | (uintptr_t)out) & 15) == 0) {
    // 64 columns a block, or fewer, down to 16, while that leaves SMs without one
    int CB = 64;
    while (CB > 16 && (CB / 2 >= D || (long)R * H * ((D + CB - 1) / CB) < 132)) CB /= 2;
    const int c4 = CB / 4, rows = (D * c4 + DS_THREADS - 1) / DS_THREADS;
    const dim3 single((D + CB - 1) / CB, H, R);
#define DS_SINGLE(N)                                                                                                             \
  qb_launch(delta_single_kernel<N>, single, DS_THREADS, 0, stream, proj, proj_stride, r_off, k_off, v_off, a_off, wpre, a_bias, w_bias,  \
                                                            state, out, req_start, req_slot, H, D, c4, decay_scale, unit_eps)
    if (rows <= 2) DS_SINGLE(2);
    else if (rows <= 4) DS_SINGLE(4);
    else DS_SINGLE(8);
#undef DS_SINGLE
    QB_LAUNCH_CHECK();
    return 0;
  }
  const size_t n = (size_t)T * H * D;
  float *w_s = scratch, *au_s = scratch + n, *u_s = scratch + 2 * n;
  const long warps = (long)T * H;
  delta_prep_kernel<<<(int)((warps + 3) / 4), 128, 0, stream>>>(proj, proj_stride, k_off, a_off, wpre, a_bias, w_bias,
                                                              w_s, au_s, u_s, T, H, D, decay_scale, unit_eps);
  QB_LAUNCH_CHECK();
  // columns a block: all of them (at most DR_MAX_COLS) unless that leaves most SMs idle; then fewer, down to 16
  // where requests bring portions (the block's threads also fetch the chunks) and down to 4 where every request
  // brings one token (the state's bytes are what counts, spread over all SMs); a multiple of 4: whole warps
  const int min_cols = T > R ? 16 : 4;
  int splits = (D + DR_MAX_COLS - 1) / DR_MAX_COLS;
  while ((long)R * H * splits < 132 && (D + 2 * splits - 1) / (2 * splits) >= min_cols) splits *= 2;
  int cols = (D + splits - 1) / splits;
  cols = (cols + 3) / 4 * 4;
  splits = (D + cols - 1) / cols;
  const int threads = cols * DR_LANES;
  const int rpt = D <= 32 ? 4 : D <= 64 ? 8 : D <= 128 ? 16 : 32;
  const int dp = rpt * DR_LANES;
  const int chunk = dp <= 128 ? 16 : 8;
  const size_t smem = (size_t)12 * chunk * dp * sizeof(float);
  dim3 grid(R, H, splits);
#define DR_LAUNCH(N)                                                                                       \
  do {                                                                                                     \
    auto kern = delta_rule_kernel<N>;                                                                      \
    if (smem > 48 * 1024) {                                                                                \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
      if (e != cudaSuccess) return (int)e;                                                                 \
    }                                                                                                      \
    kern<<<grid, threads, smem, stream>>>(proj, proj_stride, r_off, k_off, v_off, w_s, au_s, u_s, state,   \
                                          out, req_start, req_slot, H, D, cols, chunk);                    \
  } while (0)
  if (rpt == 4) DR_LAUNCH(4);
  else if (rpt == 8) DR_LAUNCH(8);
  else if (rpt == 16) DR_LAUNCH(16);
  else DR_LAUNCH(32);
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
