// Generalized delta rule with a decay per key channel: a recurrence over time whose state is a matrix
// S [key channel i, value channel j] per (request, head), float32, kept in the request's state slot.
//
//   u   = k / sqrt(sum(k^2) + unit_eps)                       (unit key of the head)
//   w   = exp(-decay_scale * sigmoid(wpre + w_bias))          (decay per key channel)
//   a   = sigmoid(apre + a_bias)                              (removal rate per key channel)
//   S_t = diag(w) S_{t-1} - (a * u) (u^T S_{t-1}) + k v^T     (both terms read the old state)
//   o_t = S_t^T r
//
// A column j of S never meets another column.  Sixteen lanes share one: lane p has its rows p + 16 n.  Its part of u^T S (and of the output)
// is two sums, over the rows of even and of odd n in the order of n, added up; the sixteen parts meet two by two (lanes 8, 4, 2, 1 apart).
// Both kernels below do exactly these operations, so a position's numbers depend neither on the cut nor on the batch, not even by rounding.
// (Portions once ran in chunks of 16 tokens as products, 270 us for the prompt below where the chain of that time took 403; their outputs were
// 1.7e-7 off float64 against 1.1e-7 here, and depended on what shared the step.)
//
// The per-head RMS norm with gain and gate that follows is a kernel of the common unit (norm_embed.cu).
#include "common.cuh"

constexpr int DR_LANES = 16;  // lanes that share a column
constexpr int DR_ARRAYS = 5;  // of a (token, head): u, w, a*u, k, r

// Two float32 numbers in one 64-bit register: the halves of a packed operation round as the operations of one number do.
typedef unsigned long long dr_pair;
__device__ __forceinline__ dr_pair dr_pack(float a, float b) {
  dr_pair v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void dr_unpack(dr_pair v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ dr_pair dr_fma(dr_pair a, dr_pair b, dr_pair c) {
  dr_pair v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ dr_pair dr_mul(dr_pair a, dr_pair b) {
  dr_pair v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

// What a token does to two rows of a column: k v + (w s + a u (-dot)).
__device__ __forceinline__ dr_pair dr_rows2(dr_pair w, dr_pair s, dr_pair au, dr_pair minus_dot, dr_pair k, dr_pair v) {
  return dr_fma(k, v, dr_fma(w, s, dr_mul(au, minus_dot)));
}
__device__ __forceinline__ float dr_decay(float x, float scale) { return expf(-scale * (1.f / (1.f + expf(-x)))); }
__device__ __forceinline__ float dr_rate(float x) { return 1.f / (1.f + expf(-x)); }
// 1 / |k| of a head, by one warp: the same additions wherever it is called
__device__ __forceinline__ float dr_unit(const float* k, int D, int lane, float unit_eps) {
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) ss = fmaf(k[i], k[i], ss);
  return 1.f / sqrtf(qb_warp_sum(ss) + unit_eps);
}

// ---------------------------------------------------------------------------------------------
// Portions.  A first kernel turns the projections of every (head, token) into arrays of DP floats: u, w, a*u, k, r in the order in which the
// lanes read them (row i = p + 16 (4 q + e) is number (16 q + p) 4 + e, zeros past D, so that a lane's rows are 16-byte pieces and the pieces of
// the sixteen lanes lie side by side).  A head's tokens follow one another: a chunk of them is one run of memory.
//
// The recurrence is a chain in time.  A lane group owns two columns in registers for the whole portion, a block some columns of one
// (request, head).  Chunks of 16 tokens come into shared memory by copies of a warp of their own, three ahead.  One portion alone is bound by the
// chain of a token: two packed multiply-adds, four exchanges (29 cycles each), three more packed operations; the rows of the next token are
// read meanwhile, and the sixteen tokens' outputs are summed over the lanes together (16 exchanges a column instead of 64).  Eight lanes
// a column have one exchange less but twice the reads of shared memory, behind which the exchanges queue (281 us for the prompt below, 240 with
// sixteen; with a branch a token around the step 338).  Enough portions to fill the SMs are bound by the reads of the five arrays, which
// four columns a lane halve.  Measured on a B200, chain and preparation, with eight lanes a column / with this: one portion of 2,048 tokens, 32
// heads of 64, 378 / 298 us, 8 of 512 355 / 329, 16 heads of 128 588 / 410 and 574 / 502, 8 heads of 256, 300 tokens, 172 / 114, 23 single
// tokens beside 512 236 / 160.
// ---------------------------------------------------------------------------------------------
constexpr int DR_MAX_COLS = 32, DR_CHUNK_FLOATS = 16 * DR_ARRAYS * 64, DR_STAGE_FLOATS = DR_CHUNK_FLOATS + 16 * DR_MAX_COLS, DR_STAGES = 4;

template <int RPT>
__global__ void __launch_bounds__(128)
delta_prep_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int a_off, const float* __restrict__ wpre,
                  const float* __restrict__ a_bias, const float* __restrict__ w_bias, float* __restrict__ scratch, int T, int H, int D,
                  float decay_scale, float unit_eps) {
  constexpr int DP = DR_LANES * RPT, N = DP / 32;
  const int lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= (long)T * H) return;
  const int t = (int)(wid / H), h = (int)(wid % H);
  const float* row = proj + (size_t)t * proj_stride + (size_t)h * D;
  float k[N], a[N], w[N], r[N], ab[N], wb[N];              // all reads before the first use
#pragma unroll
  for (int x = 0; x < N; ++x) {
    const int at = lane + 32 * x, i = ((at >> 2) & 15) + DR_LANES * ((at & 3) + 4 * (at >> 6));
    const bool in = i < D;
    k[x] = in ? row[k_off + i] : 0.f;
    a[x] = in ? row[a_off + i] : 0.f;
    w[x] = in ? wpre[(size_t)wid * D + i] : 0.f;
    r[x] = in ? row[r_off + i] : 0.f;
    ab[x] = in ? a_bias[h * D + i] : 0.f;
    wb[x] = in ? w_bias[h * D + i] : 0.f;
  }
  const float inv = dr_unit(row + k_off, D, lane, unit_eps);
  float* to = scratch + ((size_t)h * T + t) * DR_ARRAYS * DP;
#pragma unroll
  for (int x = 0; x < N; ++x) {
    const int at = lane + 32 * x, i = ((at >> 2) & 15) + DR_LANES * ((at & 3) + 4 * (at >> 6));
    const bool in = i < D;
    const float u = k[x] * inv;
    to[at] = u;                                              // (past D: k is zero)
    to[DP + at] = in ? dr_decay(w[x] + wb[x], decay_scale) : 0.f;
    to[2 * DP + at] = in ? dr_rate(a[x] + ab[x]) * u : 0.f;
    to[3 * DP + at] = k[x];
    to[4 * DP + at] = r[x];
  }
}

// The sums over the sixteen lanes of N values each, N at most 16: lane p then holds the value dr_first<N>(p) (lanes that differ in their lower
// bits only, those that N does not use, hold the same).
template <int N>
__device__ __forceinline__ void dr_sum_lanes(float (&x)[N], int p) {
  int n = N;
#pragma unroll
  for (int d = DR_LANES / 2; d > 0; d >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool upper = p & d;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i >= n) break;
        const float give = upper ? x[i] : x[i + n], keep = upper ? x[i + n] : x[i];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, give, d);
      }
    } else {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], d);
    }
  }
}
template <int N>
__device__ __forceinline__ int dr_first(int p) {
  int first = 0, n = N;
#pragma unroll
  for (int d = DR_LANES / 2; n > 1; d >>= 1) {
    n >>= 1;
    first += p & d ? n : 0;
  }
  return first;
}

__device__ __forceinline__ unsigned dr_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool dr_done(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: false when the limit (iterations and 0.2 s) is reached or, where there is a flag, another warp gave up.
__device__ __forceinline__ bool dr_wait(unsigned bar, unsigned parity, volatile int* abort_flag) {
  unsigned long long t0 = 0;
  for (unsigned it = 0; it < 4000000u; ++it) {
    if (dr_done(bar, parity)) return true;
    if ((it & 63u) == 63u) {
      if (abort_flag != nullptr && *abort_flag) return false;
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > 200000000ull) break;
    }
  }
  if (abort_flag != nullptr) *abort_flag = 1;
  return false;
}

// RPT: rows of a column a lane holds (D <= 16 RPT); C: columns a lane; U: tokens whose outputs are summed together.  Four warps walk the
// tokens, one more brings them.
template <int RPT, int C, int U>
__global__ void __launch_bounds__(160, C == 4 ? 2 : 1)
delta_rule_kernel(const float* __restrict__ proj, int proj_stride, int v_off, const float* __restrict__ scratch, float* __restrict__ state,
                  float* __restrict__ out, const int* __restrict__ req_start, const int* __restrict__ req_slot, int T, int H, int D, int* status) {
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) unsigned long long s_full[DR_STAGES], s_empty[DR_STAGES];
  __shared__ int s_abort;
  constexpr int DP = DR_LANES * RPT, PER = DR_ARRAYS * DP, P = RPT / 2, W = 4;
  constexpr int CHUNK = DR_CHUNK_FLOATS / PER, COLS = 2 * W * C;    // 16 tokens of heads up to 64, fewer of larger ones
  const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int p = tid % DR_LANES, col0 = blockIdx.z * COLS, jj = tid / DR_LANES * C, j = col0 + jj;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (t0 >= t1) return;
  const unsigned sm0 = dr_smem(sm);
  const int n_all = t1 - t0, chunks = (n_all + CHUNK - 1) / CHUNK;
  volatile int* abort_flag = &s_abort;
  if (tid == 0) {
    for (int b = 0; b < DR_STAGES; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(dr_smem(&s_full[b])));       // the run of scratch, and each lane's copies
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(dr_smem(&s_empty[b])), "r"(W));
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid >= 32 * W) {
    // ---- the warp that brings the tokens.  A stage: [CHUNK][PER] in one copy, then v [CHUNK][COLS], 4 bytes a copy (columns start
    // anywhere; past D zeros)
    const int lane = tid & 31;
    const float* from = scratch + ((size_t)h * T + t0) * PER;
    const float* v_from = proj + (size_t)t0 * proj_stride + v_off + (size_t)h * D + col0;
    int c = 0;
    for (; c < chunks; ++c) {
      const int b = c % DR_STAGES, n = min(CHUNK, n_all - c * CHUNK);
      if (c >= DR_STAGES && !__all_sync(0xffffffffu, dr_wait(dr_smem(&s_empty[b]), (unsigned)(c / DR_STAGES - 1) & 1u, abort_flag))) break;
      const unsigned to = sm0 + 4 * b * DR_STAGE_FLOATS, bar = dr_smem(&s_full[b]);
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(4 * n * PER) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(to), "l"(from + (size_t)c * DR_CHUNK_FLOATS), "r"(4 * n * PER), "r"(bar) : "memory");
      }
#pragma unroll 4
      for (int i = lane; i < n * COLS; i += 32) {
        const int tt = i / COLS, x = i % COLS;
        const bool in = col0 + x < D;
        const float* v = in ? v_from + (size_t)(c * CHUNK + tt) * proj_stride + x : proj;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4 * (CHUNK * PER + i)), "l"(v), "r"(in ? 4 : 0) : "memory");
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    }
    // whichever warp gives up, the copies on their way land before the block leaves its shared memory
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int x = max(0, c - DR_STAGES); x < c; ++x) dr_wait(dr_smem(&s_full[x % DR_STAGES]), (unsigned)(x / DR_STAGES) & 1u, nullptr);
  } else {
    float* S = state + ((size_t)req_slot[r] * H + h) * D * D + j;
    auto held = [&](int n, int e) { return j + e < D && p + DR_LANES * n < D; };
    auto cell = [&](int n, int e) { return held(n, e) ? S[(size_t)(p + DR_LANES * n) * D + e] : 0.f; };
    dr_pair col[C][P];
#pragma unroll
    for (int e = 0; e < C; ++e)
#pragma unroll
      for (int i = 0; i < P; ++i) col[e][i] = dr_pack(cell(2 * i, e), cell(2 * i + 1, e));
    struct Token {
      dr_pair u[P], w[P], au[P], k[P], r[P];
      float v[C];
    };
    // shared-memory reads that stay where they are written, before the exchanges of the token in work (the compiler put them behind: 368 us)
    auto rows = [&](unsigned a, dr_pair (&x)[P]) {               // this lane's rows of one array
#pragma unroll
      for (int q = 0; q < P / 2; ++q)
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x[2 * q]), "=l"(x[2 * q + 1]) : "r"(a + 16 * (q * DR_LANES)));
    };
    auto read = [&](unsigned a, unsigned v, Token& t) {
      rows(a, t.u); rows(a + 8 * DP, t.au); rows(a + 4 * DP, t.w); rows(a + 12 * DP, t.k); rows(a + 16 * DP, t.r);
      if constexpr (C == 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(t.v[0]), "=f"(t.v[1]) : "r"(v));
      else asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(t.v[0]), "=f"(t.v[1]), "=f"(t.v[2]), "=f"(t.v[3]) : "r"(v));
    };
    auto step = [&](const Token& t, float (&o)[C]) {             // this lane's part of the output
      float dot[C];
#pragma unroll
      for (int e = 0; e < C; ++e) {
        dr_pair sum = 0;
#pragma unroll
        for (int i = 0; i < P; ++i) sum = dr_fma(t.u[i], col[e][i], sum);
        float a, b;
        dr_unpack(sum, a, b);
        dot[e] = a + b;
      }
#pragma unroll
      for (int d = DR_LANES / 2; d > 0; d >>= 1)
#pragma unroll
        for (int e = 0; e < C; ++e) dot[e] += __shfl_xor_sync(0xffffffffu, dot[e], d);
#pragma unroll
      for (int e = 0; e < C; ++e) {
        const dr_pair minus = dr_pack(-dot[e], -dot[e]), v = dr_pack(t.v[e], t.v[e]);
        dr_pair sum = 0;
#pragma unroll
        for (int i = 0; i < P; ++i) col[e][i] = dr_rows2(t.w[i], col[e][i], t.au[i], minus, t.k[i], v);
#pragma unroll
        for (int i = 0; i < P; ++i) sum = dr_fma(t.r[i], col[e][i], sum);
        float a, b;
        dr_unpack(sum, a, b);
        o[e] = a + b;
      }
    };
    float* to = out + ((size_t)t0 * H + h) * D + j;
    const size_t next = (size_t)H * D;
    bool ok = true;
    for (int c = 0; c < chunks; ++c) {
      const int b = c % DR_STAGES;
      ok = __all_sync(0xffffffffu, dr_wait(dr_smem(&s_full[b]), (unsigned)(c / DR_STAGES) & 1u, abort_flag));
      if (!ok) break;
      unsigned a = sm0 + 4 * b * DR_STAGE_FLOATS, v = a + 4 * (CHUNK * PER + jj);
      a += 16 * p;
      const int n = min(CHUNK, n_all - c * CHUNK);
      Token now;
      read(a, v, now);
      int tt = 0;
#pragma unroll 1
      for (; tt + U <= n; tt += U) {          // no branch inside: the next token's rows are read during this one's exchanges
        float o[C][U];
#pragma unroll
        for (int x = 0; x < U; ++x) {
          Token ahead;
          read(a + 4 * (x + 1) * PER, v + 4 * (x + 1) * COLS, ahead);      // behind the last token: whatever lies there, not used
          float part[C];
          step(now, part);
#pragma unroll
          for (int e = 0; e < C; ++e) o[e][x] = part[e];
          now = ahead;
        }
        a += 4 * U * PER;
        v += 4 * U * COLS;
        const int first = dr_first<U>(p);
#pragma unroll
        for (int e = 0; e < C; ++e) {
          dr_sum_lanes<U>(o[e], p);
          if (p % (DR_LANES / U) == 0 && j + e < D) to[(size_t)first * next + e] = o[e][0];
        }
        to += U * next;
      }
#pragma unroll 1
      for (; tt < n; ++tt) {                  // the portion's last tokens
        float o[C];
        read(a, v, now);
        a += 4 * PER;
        v += 4 * COLS;
        step(now, o);
#pragma unroll
        for (int e = 0; e < C; ++e) {
          float one[1] = {o[e]};
          dr_sum_lanes<1>(one, p);
          if (p == 0 && j + e < D) to[e] = one[0];
        }
        to += next;
      }
      __syncwarp();
      if ((tid & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dr_smem(&s_empty[b])) : "memory");
    }
    if (ok) {
#pragma unroll
      for (int e = 0; e < C; ++e)
#pragma unroll
        for (int i = 0; i < P; ++i) {
          float x, y;
          dr_unpack(col[e][i], x, y);
          if (held(2 * i, e)) S[(size_t)(p + DR_LANES * 2 * i) * D + e] = x;
          if (held(2 * i + 1, e)) S[(size_t)(p + DR_LANES * (2 * i + 1)) * D + e] = y;
        }
    }
  }
  // behind the last wait of every warp: whoever gave up, the failure is seen (outputs behind it and the state are not written)
  __syncthreads();
  if (tid == 0 && s_abort) qb_set_status(status, QB_STATUS_WAIT_TIMEOUT, r, 9);
}

// ---------------------------------------------------------------------------------------------
// Steps in which every request brings one token: preparation and recurrence in one launch.  A thread takes four columns of its rows, so
// that S is read and written in 16-byte pieces that are asked for before anything else; a warp takes 16 columns, a block 16 to 64 of one
// (request, head).  Bound by the chain of the unit key's sum and two column sums.  8 tokens, 32 heads of 64 (8.4 MB of state): 10.4 us
// as two launches with the columns of S read a float at a time, 4.5 us with this; 64 tokens 51 and 19.
// ---------------------------------------------------------------------------------------------
constexpr int DS_MAX_DIM = 128;

template <int RPT>
__global__ void __launch_bounds__(128, RPT == 4 ? 6 : 3)
delta_single_kernel(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                    const float* wpre, const float* a_bias, const float* w_bias,
                    float* state, float* __restrict__ out, const int* req_start,
                    const int* req_slot, int H, int D, int cols, float decay_scale, float unit_eps, int early) {
  if (!early) qb_follow();
  constexpr int DP = DR_LANES * RPT;
  __shared__ float s_u[DP], s_w[DP], s_au[DP], s_k[DP], s_r[DP];
  const int tid = threadIdx.x, lane = tid & 31, h = blockIdx.y, r = blockIdx.z;
  const int p = lane >> 2, c = (tid >> 5) * 16 + (lane & 3) * 4, j = blockIdx.x * cols + c;
  const int t0 = req_start[r], t1 = req_start[r + 1];
  if (!early && t0 >= t1) return;
  float* S = state + ((size_t)req_slot[r] * H + h) * D * D + j;
  const bool owns = c < cols && j < D && t0 < t1;      // other warps help with the preparation
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // four columns; a lane stands for the lanes p (v = 0) and p + 8 (v = 1) of the kernel for portions, whose parts meet first
  constexpr int P = RPT / 2;
  dr_pair st[4][2][P];
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int x = p + 8 * v + DR_LANES * 2 * i, y = x + DR_LANES;
      const float4 a = x < D && owns ? *reinterpret_cast<const float4*>(S + (size_t)x * D) : zero;
      const float4 b = y < D && owns ? *reinterpret_cast<const float4*>(S + (size_t)y * D) : zero;
      st[0][v][i] = dr_pack(a.x, b.x); st[1][v][i] = dr_pack(a.y, b.y); st[2][v][i] = dr_pack(a.z, b.z); st[3][v][i] = dr_pack(a.w, b.w);
    }
  // the state is on its way while the launch before ends
  if (early) qb_follow();
  if (t0 >= t1) return;
  auto over_lanes = [&](const dr_pair (&sum)[4][2], float (&x)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a, b, c, d;
      dr_unpack(sum[e][0], a, b);
      dr_unpack(sum[e][1], c, d);
      x[e] = (a + b) + (c + d);
    }
#pragma unroll
    for (int o = 16; o > 2; o >>= 1)
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] += __shfl_xor_sync(0xffffffffu, x[e], o);
  };
  auto two = [&](const float* a, int v, int i) { return dr_pack(a[p + 8 * v + DR_LANES * 2 * i], a[p + 8 * v + DR_LANES * (2 * i + 1)]); };
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
    const float ve[4] = {v.x, v.y, v.z, v.w};
    dr_pair sum[4][2] = {};
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const dr_pair u = two(s_u, w, i);
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e][w] = dr_fma(u, st[e][w][i], sum[e][w]);
      }
    float dot[4], o[4];
    over_lanes(sum, dot);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e][0] = sum[e][1] = 0;
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const dr_pair w = two(s_w, z, i), au = two(s_au, z, i), k = two(s_k, z, i), rr = two(s_r, z, i);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          st[e][z][i] = dr_rows2(w, st[e][z][i], au, dr_pack(-dot[e], -dot[e]), k, dr_pack(ve[e], ve[e]));
          sum[e][z] = dr_fma(rr, st[e][z][i], sum[e][z]);
        }
      }
    over_lanes(sum, o);
    if (p == 0 && owns) *reinterpret_cast<float4*>(out + ((size_t)t * H + h) * D + j) = make_float4(o[0], o[1], o[2], o[3]);
    if (t + 1 < t1) __syncthreads();
  }
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int i = 0; i < P; ++i) {
      float a[4], b[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) dr_unpack(st[e][v][i], a[e], b[e]);
      const int x = p + 8 * v + DR_LANES * 2 * i, y = x + DR_LANES;
      if (x < D && owns) *reinterpret_cast<float4*>(S + (size_t)x * D) = make_float4(a[0], a[1], a[2], a[3]);
      if (y < D && owns) *reinterpret_cast<float4*>(S + (size_t)y * D) = make_float4(b[0], b[1], b[2], b[3]);
    }
}

static int dr_rows(int D) { return D <= 64 ? 4 : D <= 128 ? 8 : 16; }

// Floats of scratch that a step wants.
extern "C" long long qb_delta_rule_scratch(int T, int H, int D) {
  return T <= 0 || H <= 0 || D <= 0 || D > 256 ? 0 : (long long)T * H * DR_ARRAYS * DR_LANES * dr_rows(D);
}

// scratch: qb_delta_rule_scratch floats, on 16 bytes.  early: the two launches before this one write neither the state nor req_start and
// req_slot (a step of single tokens then reads them before the launch before it has ended).
extern "C" int qb_delta_rule(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                             const float* wpre, const float* a_bias, const float* w_bias, float* state,
                             float* out, float* scratch, const int* req_start, const int* req_slot, int R,
                             int T, int H, int D, float decay_scale, float unit_eps, int early, int* status, cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  if (D <= 0 || D > 256 || H <= 0) return QB_ERR_UNSUPPORTED;
  const int rpt = dr_rows(D), dp = rpt * DR_LANES;
  if (T == R && D % 4 == 0 && D <= DS_MAX_DIM && H <= 65535 && R <= 65535 && (((uintptr_t)state | (uintptr_t)out) & 15) == 0) {
    // 64 columns a block, or fewer, down to 16, while that leaves SMs without one
    int CB = 64;
    while (CB > 16 && (CB / 2 >= D || (long)R * H * ((D + CB - 1) / CB) < 132)) CB /= 2;
    const dim3 single((D + CB - 1) / CB, H, R);
#define DS_SINGLE(N)                                                                                                                \
  qb_launch(delta_single_kernel<N>, single, 128, 0, stream, proj, proj_stride, r_off, k_off, v_off, a_off, wpre, a_bias, w_bias, \
            state, out, req_start, req_slot, H, D, CB, decay_scale, unit_eps, early)
    if (rpt == 4) DS_SINGLE(4);
    else DS_SINGLE(8);
#undef DS_SINGLE
    QB_LAUNCH_CHECK();
    return 0;
  }
  if (((uintptr_t)scratch & 15) != 0) return QB_ERR_BAD_ARG;
  const long warps = (long)T * H;
#define DR_PREP(N)                                                                                                              \
  delta_prep_kernel<N><<<(int)((warps + 3) / 4), 128, 0, stream>>>(proj, proj_stride, r_off, k_off, a_off, wpre, a_bias, w_bias, \
                                                                   scratch, T, H, D, decay_scale, unit_eps)
  if (rpt == 4) DR_PREP(4);
  else if (rpt == 8) DR_PREP(8);
  else DR_PREP(16);
#undef DR_PREP
  QB_LAUNCH_CHECK();
  // four columns a lane, 32 a block (heads of at most 128, for the registers), or two and 16 where that leaves SMs idle
  const bool wide = rpt <= 8 && D > 16 && (long)R * H * ((D + 31) / 32) >= 132;
  const int cols = wide ? 32 : 16;
  const size_t smem = ((size_t)DR_STAGES * DR_STAGE_FLOATS + DR_ARRAYS * dp) * sizeof(float);      // (reads go a token past the end)
  dim3 grid(R, H, (D + cols - 1) / cols);
#define DR_LAUNCH(N, C, U)                                                                                                     \
  do {                                                                                                                         \
    auto kern = delta_rule_kernel<N, C, U>;                                                                                    \
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                  \
    if (e != cudaSuccess) return (int)e;                                                                                       \
    kern<<<grid, 160, smem, stream>>>(proj, proj_stride, v_off, scratch, state, out, req_start, req_slot, T, H, D, status);    \
  } while (0)
  if (rpt == 4 && wide) DR_LAUNCH(4, 4, 8);
  else if (rpt == 4) DR_LAUNCH(4, 2, 16);
  else if (rpt == 8 && wide) DR_LAUNCH(8, 4, 4);
  else if (rpt == 8) DR_LAUNCH(8, 2, 8);
  else DR_LAUNCH(16, 2, 4);
#undef DR_LAUNCH
  QB_LAUNCH_CHECK();
  return 0;
}

// out[t, c] = tanh(x[t, off + c]) for c < n, in the activation dtype (the inner activation of a
// low-rank pair of projections whose first product sits inside a wider fused product).
template <typename O>
__global__ void tanh_cols_kernel(const float* x, int x_stride, int off, O* __restrict__ out,
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

// out[t, n] = sum_l a(tanh(x[t, off + l])) w[n, l], a: rounding to bfloat16: the inner activation of a low-rank pair of projections and its
// outer product, for steps of few rows, whose two launches (4.5 us in a step of 8 requests) this is one of.  The L products of an output
// are exact in float64 and are added there, so that the result is rounded once.
template <int L>
__global__ void __launch_bounds__(128) tanh_product_kernel(const float* x, int x_stride, int off, const __nv_bfloat16* w,
                                                           float* __restrict__ out, int n, int N) {
  __shared__ float s_in[L];
  const int row = blockIdx.x * 128 + threadIdx.x;
  __nv_bfloat16 wr[L];
  qb_follow();
#pragma unroll
  for (int l = 0; l < L; ++l) wr[l] = row < N && l < n ? w[(size_t)row * n + l] : __float2bfloat16_rn(0.f);
  const int t = blockIdx.y;
  for (int i = threadIdx.x; i < n; i += 128) s_in[i] = __bfloat162float(__float2bfloat16_rn(tanhf(x[(size_t)t * x_stride + off + i])));
  __syncthreads();
  if (row >= N) return;
  double sum = 0.0;
#pragma unroll
  for (int l = 0; l < L; ++l)
    if (l < n) sum += (double)s_in[l] * (double)__bfloat162float(wr[l]);
  out[(size_t)t * N + row] = (float)sum;
}

extern "C" int qb_tanh_product(const float* x, int x_stride, int off, const void* w, float* out, int T, int n, int N, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  if (n <= 0) return QB_ERR_BAD_ARG;
  if (T > 32 || n > 64) return QB_ERR_UNSUPPORTED;
  const dim3 grid((N + 127) / 128, T);
  if (n <= 16) qb_launch(tanh_product_kernel<16>, grid, 128, 0, stream, x, x_stride, off, (const __nv_bfloat16*)w, out, n, N);
  else qb_launch(tanh_product_kernel<64>, grid, 128, 0, stream, x, x_stride, off, (const __nv_bfloat16*)w, out, n, N);
  QB_LAUNCH_CHECK();
  return 0;
}
