// q/k RMSNorm + partial rotary position encoding + query temperature + write of K and V into the paged cache,
// one kernel.
//
// Input is a row of a fused projection, [q | k | v | anything else] (row_stride elements), of every token of the
// step; a layer that reads another layer's cache has rows [q | anything else] (has_kv = 0).  For each token:
//   q, k  <- RMSNorm (none | over all heads of the row | per head), float32
//            (src/quanta/minimax/model_m3.py:15-17 / src/quanta/minimax/attention.py:172-182)
//   q, k  <- rotation of the first `rd` dims of each head, pair j using position axis pair_axis[j] and angle
//            float(pos) * inv_freq[j]; pair j is the dims (j, j + rd/2)  (src/quanta/minimax/model_m3.py:83-96), or
//            with `interleaved` the neighbours (2j, 2j + 1)
//   q     <- q * (1 + temp_coef * ln(floor((pos + 1) / temp_every) + 1))     (temp_every > 0: a query
//            temperature that grows with the position, float32)
//   q     <- q * head_scale[head]          (head_scale: a float32 number per q head that multiplies the head's
//            scores; null for none)
//   v     <- (1 - lambda) v + lambda v_first      (v_first: float32 values [T, nkv * vd] that an earlier layer left for
//            the same tokens, lambda one number on the device; v_export: this layer leaves its own values there)
//   v     =  the projected k before norm and rotation (tied_v: the rows are [q | k | anything else], vd == hd)
//   q     -> q_out [T, nq, hd];  k -> pages [page, kv_head, slot, hd], v -> pages [page, kv_head, slot, vd]
//            through the block table (keys and values may have different head sizes)
// The rows may be float32 accumulators of the projection while q and the cache are in the activation dtype, and a
// bias (float32, laid out like the row's [q | k | v]) may be added first.  A per-head norm may have no gains.
// One rounding to the activation dtype, at the store.  One block per token.
#include "common.cuh"

#define NORM_NONE 0
#define NORM_PER_LAYER 1
#define NORM_PER_HEAD 2

template <typename IN, typename A>
__global__ void qknorm_rope_write_kernel(
    const IN* __restrict__ qkv, int row_stride, A* __restrict__ q_out, A* __restrict__ k_cache, A* __restrict__ v_cache,
    const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w, int norm_kind, float eps,
    const float* __restrict__ inv_freq, const int* __restrict__ pair_axis,
    const int* __restrict__ positions, int n_axes, const int* __restrict__ tok_pos,
    const int* __restrict__ tok_req, const int* __restrict__ block_table, int bt_stride, int T, int nq,
    int nkv_all, int hd, int vd, int has_kv, int tied_v, int rd, int interleaved, float temp_coef, int temp_every, int page_size, int num_pages,
    int vec, const float* __restrict__ bias, const float* __restrict__ v_first, const float* __restrict__ v_lambda,
    float* __restrict__ v_export, const float* __restrict__ head_scale, int* status) {
  extern __shared__ float smem[];
  const int t = blockIdx.x;
  if (t >= T) return;
  const int nkv = has_kv ? nkv_all : 0;
  const int qn = nq * hd, kn = nkv * hd, vn = nkv * vd;
  float* buf = smem;                 // [qn + kn]  q then k
  float* cs = buf + qn + kn;         // [rd/2] cos, [rd/2] sin
  float* scratch = cs + rd;          // 32 + (nq + nkv) head statistics
  float* head_r = scratch + 32;
  const IN* row = qkv + (size_t)t * row_stride;
  const int half = rd / 2;
  // Where this token's K and V go is a chain of three dependent loads (position, request, page id), and the
  // norm gains come from memory that the layer's expert weights have pushed out of L2: both are asked for
  // now, so that their latency passes under the phases below instead of after them.
  int pos = 0, page = -1;
  if (k_cache != nullptr || temp_every > 0) pos = tok_pos[t];
  if (k_cache != nullptr) page = block_table[(size_t)tok_req[t] * bt_stride + pos / page_size];
  const int n_chunks = vec ? (qn + kn) / 8 : 0;
  float w_first[8];                  // the gains of this thread's first chunk (NORM_PER_LAYER)
  if (norm_kind == NORM_PER_LAYER && (int)threadIdx.x < n_chunks) {
    const int i = threadIdx.x * 8;
    QbVec8<float>::load(i < qn ? q_norm_w + i : k_norm_w + (i - qn), w_first);
  }

  if (vec) {
    // 16-byte loads, all of a thread's loads issued before their first use
#pragma unroll 4
    for (int c = threadIdx.x; c < n_chunks; c += blockDim.x) {
      float v[8];
      QbVec8<IN>::load(row + c * 8, v);
      if (bias != nullptr) {
        float b[8];
        QbVec8<float>::load(bias + c * 8, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += b[e];
      }
      QbVec8<float>::store(buf + c * 8, v);
    }
  } else {
    for (int i = threadIdx.x; i < qn + kn; i += blockDim.x)
      buf[i] = qb_to_float<IN>(row[i]) + (bias != nullptr ? bias[i] : 0.f);
  }
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    const int ax = pair_axis ? pair_axis[j] : 0;
    const float ang = (float)positions[(size_t)t * n_axes + ax] * inv_freq[j];
    float s, c;
    sincosf(ang, &s, &c);
    cs[j] = c;
    cs[half + j] = s;
  }
  __syncthreads();

  if (norm_kind == NORM_PER_LAYER) {
    // a warp per head, then the heads' sums in head order: the same additions whatever the block size
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int h = warp; h < nq + nkv; h += nwarps) {
      float sh = 0.f;
      for (int d = lane; d < hd; d += 32) sh += buf[h * hd + d] * buf[h * hd + d];
      sh = qb_warp_sum(sh);
      if (lane == 0) head_r[h] = sh;
    }
    __syncthreads();
    float tq = 0.f, tk = 0.f;
    for (int h = 0; h < nq; ++h) tq += head_r[h];
    for (int h = 0; h < nkv; ++h) tk += head_r[nq + h];
    const float rq = rsqrtf(tq / (float)qn + eps), rk = rsqrtf(tk / (float)max(kn, 1) + eps);
    if (vec) {
#pragma unroll 4
      for (int c = threadIdx.x; c < n_chunks; c += blockDim.x) {
        const int i = c * 8;
        float w[8], v[8];
        if (c == (int)threadIdx.x) {
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = w_first[e];
        } else {
          QbVec8<float>::load(i < qn ? q_norm_w + i : k_norm_w + (i - qn), w);
        }
        QbVec8<float>::load(buf + i, v);
        const float r = i < qn ? rq : rk;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = w[e] * (v[e] * r);
        QbVec8<float>::store(buf + i, v);
      }
    } else {
      for (int i = threadIdx.x; i < qn + kn; i += blockDim.x)
        buf[i] = (i < qn ? q_norm_w[i] : k_norm_w[i - qn]) * (buf[i] * (i < qn ? rq : rk));
    }
    __syncthreads();
  } else if (norm_kind == NORM_PER_HEAD) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int h = warp; h < nq + nkv; h += nwarps) {
      float s = 0.f;
      for (int d = lane; d < hd; d += 32) s += buf[h * hd + d] * buf[h * hd + d];
      s = qb_warp_sum(s);
      if (lane == 0) head_r[h] = rsqrtf(s / (float)hd + eps);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < qn + kn; i += blockDim.x) {
      const int h = i / hd, d = i % hd;
      const float w = q_norm_w == nullptr ? 1.f : h < nq ? q_norm_w[d] : k_norm_w[d];
      buf[i] = w * (buf[i] * head_r[h]);
    }
    __syncthreads();
  }

  // rotation: each (head, pair) is owned by one thread
  for (int i = threadIdx.x; i < (nq + nkv) * half; i += blockDim.x) {
    const int h = i / half, j = i % half;
    const int ia = h * hd + (interleaved ? 2 * j : j), ib = interleaved ? ia + 1 : ia + half;
    const float a = buf[ia], b = buf[ib];
    const float c = cs[j], s = cs[half + j];
    buf[ia] = a * c - b * s;
    buf[ib] = b * c + a * s;
  }
  if (half > 0) __syncthreads();

  const float temp = temp_every > 0 ? 1.f + temp_coef * logf((float)((pos + 1) / temp_every) + 1.f) : 1.f;
  A* qo = q_out + (size_t)t * qn;
  if (vec) {
    for (int c = threadIdx.x; c < qn / 8; c += blockDim.x) {
      float v[8];
      QbVec8<float>::load(buf + c * 8, v);
      const float m = head_scale != nullptr ? temp * head_scale[c * 8 / hd] : temp;     // hd % 8 == 0 here
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= m;
      QbVec8<A>::store(qo + c * 8, v);
    }
  } else {
    for (int i = threadIdx.x; i < qn; i += blockDim.x)
      qo[i] = qb_from_float<A>(buf[i] * (head_scale != nullptr ? temp * head_scale[i / hd] : temp));
  }

  if (k_cache == nullptr) return;
  if (page < 0 || page >= num_pages) {
    if (threadIdx.x == 0) qb_set_status(status, QB_STATUS_BAD_PAGE, page, 2);
    return;
  }
  const int slot = pos % page_size;
  const IN* vrow = row + qn + (tied_v ? 0 : kn);
  const float* vbias = bias != nullptr ? bias + qn + (tied_v ? 0 : kn) : nullptr;
  const float lam = v_first != nullptr ? v_lambda[0] : 0.f;
  const float* vf = v_first != nullptr ? v_first + (size_t)t * vn : nullptr;
  float* vx = v_export != nullptr ? v_export + (size_t)t * vn : nullptr;
  if (vec) {
    for (int c = threadIdx.x; c < kn / 8; c += blockDim.x) {
      const int i = c * 8, h = i / hd, d = i % hd;
      float kv[8];
      QbVec8<float>::load(buf + qn + i, kv);
      QbVec8<A>::store(k_cache + (((size_t)page * nkv + h) * page_size + slot) * hd + d, kv);
    }
    for (int c = threadIdx.x; c < vn / 8; c += blockDim.x) {
      const int i = c * 8, h = i / vd, d = i % vd;
      float vv[8];
      QbVec8<IN>::load(vrow + i, vv);
      if (vbias != nullptr) {
        float b[8];
        QbVec8<float>::load(vbias + i, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) vv[e] += b[e];
      }
      if (vx != nullptr) QbVec8<float>::store(vx + i, vv);
      if (vf != nullptr) {
        float f[8];
        QbVec8<float>::load(vf + i, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) vv[e] = (1.f - lam) * vv[e] + lam * f[e];
      }
      QbVec8<A>::store(v_cache + (((size_t)page * nkv + h) * page_size + slot) * vd + d, vv);
    }
  } else {
    for (int i = threadIdx.x; i < kn; i += blockDim.x)
      k_cache[(((size_t)page * nkv + i / hd) * page_size + slot) * hd + i % hd] = qb_from_float<A>(buf[qn + i]);
    for (int i = threadIdx.x; i < vn; i += blockDim.x) {
      float v = qb_to_float<IN>(vrow[i]) + (vbias != nullptr ? vbias[i] : 0.f);
      if (vx != nullptr) vx[i] = v;
      if (vf != nullptr) v = (1.f - lam) * v + lam * vf[i];
      v_cache[(((size_t)page * nkv + i / vd) * page_size + slot) * vd + i % vd] = qb_from_float<A>(v);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The same for heads of 128: a warp takes a head, four elements a lane, and keeps its HPW heads of the token in registers from the
// load to the store (the kernel above passes every row through shared memory four times).  Pairs (j, j + rd/2) meet by a shuffle,
// neighbours lie in one lane.  One barrier.  Bound by one wait for memory for few tokens and by instructions for many (some 90 a
// head; blocks that walk tokens with the next row and the gains at hand were slower, 212 us for 12,800 tokens, for the warps
// they cost).  Measured on a B200 with 48 + 8 + 8 heads in bfloat16 and a norm over all heads: one token 7.7 -> 4.6 us, 64 tokens
// 7.7 -> 4.7, 536 tokens 13.4 -> 8.9, 12,800 tokens (420 MB) 248 -> 165 us; 16 + 4 heads from float32 with biases, neighbours turned: 16 tokens 4.8 -> 2.9 us,
// 4,876 tokens 37 -> 16 us.
// ---------------------------------------------------------------------------------------------
template <typename T> struct Four;
template <> struct Four<float> {
  __device__ static __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
  __device__ static __forceinline__ void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};
template <> struct Four<__nv_bfloat16> {
  __device__ static __forceinline__ float4 load(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
  }
  __device__ static __forceinline__ void store(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
};

struct RopeArgs {
  int row_stride, norm_kind, n_axes, bt_stride, nq, nkv, tied_v, rd, interleaved, temp_every, page_size, page_shift, num_pages;
  float eps, temp_coef;
  const float *q_norm_w, *k_norm_w, *inv_freq, *bias, *v_first, *v_lambda, *head_scale;
  const int *pair_axis, *positions, *tok_pos, *tok_req, *block_table;
  float* v_export;
  int* status;
};

constexpr int ROPE_HD = 128;

// the multiply-adds of both kernels below, written out, so that they round alike
__device__ __forceinline__ float squares(float4 v) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.x, v.x, v.y * v.y))); }
// c x + s o
__device__ __forceinline__ float4 turned(float4 x, float4 c, float4 o, float4 s) {
  return make_float4(fmaf(x.x, c.x, o.x * s.x), fmaf(x.y, c.y, o.y * s.y), fmaf(x.z, c.z, o.z * s.z), fmaf(x.w, c.w, o.w * s.w));
}
// neighbours (x, y) and (z, w) by two angles
__device__ __forceinline__ float4 turned_pairs(float4 x, float c, float s, float c2, float s2) {
  return make_float4(fmaf(x.x, c, -(x.y * s)), fmaf(x.y, c, x.x * s), fmaf(x.z, c2, -(x.w * s2)), fmaf(x.w, c2, x.z * s2));
}
__device__ __forceinline__ float4 negated(float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); }

template <typename IN, typename A, int HPW>
__global__ void __launch_bounds__(HPW == 2 ? 1024 : 512, HPW == 2 ? 1 : 2)
qknorm_rope_heads_kernel(const IN* qkv, A* __restrict__ q_out, A* __restrict__ k_cache, A* __restrict__ v_cache,
                         const RopeArgs a) {
  qb_follow();
  __shared__ __align__(16) float s_cos[ROPE_HD / 2], s_sin[ROPE_HD / 2];
  __shared__ float s_sum[32 * HPW];
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int nq = a.nq, nk = nq + a.nkv, n = nk + (a.tied_v ? 0 : a.nkv), half = a.rd / 2, d = lane * 4;
  const bool writes = k_cache != nullptr, normed = a.norm_kind != NORM_NONE, gained = normed && a.q_norm_w != nullptr;
  const IN* row = qkv + (size_t)t * a.row_stride + d;
  int pos = 0, page = -1;                // asked for first: a chain of dependent loads
  if (writes || a.temp_every > 0) pos = a.tok_pos[t];
  auto gains = [&](int h) {              // of a q or k head
    const float* g = h < nq ? a.q_norm_w : a.k_norm_w;
    return Four<float>::load(g + (a.norm_kind == NORM_PER_LAYER ? (h < nq ? h : h - nq) * ROPE_HD : 0) + d);
  };
  // few tokens: the gains come from memory that the layer's weights have pushed out of L2 and are asked for now; many: from L1
  constexpr bool EARLY = HPW == 2;
  float4 v[HPW], w[EARLY ? HPW : 1];
#pragma unroll
  for (int i = 0; i < HPW; ++i) {
    const int h = warp + i * warps;
    v[i] = h < n ? Four<IN>::load(row + h * ROPE_HD) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (EARLY && gained && h < nk) w[EARLY ? i : 0] = gains(h);
  }
  if (writes) {
    const int nth = a.page_shift >= 0 ? pos >> a.page_shift : pos / a.page_size;
    page = a.block_table[(size_t)a.tok_req[t] * a.bt_stride + nth];
  }
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    const int ax = a.pair_axis ? a.pair_axis[j] : 0;
    const float ang = (float)a.positions[(size_t)t * a.n_axes + ax] * a.inv_freq[j];
    sincosf(ang, &s_sin[j], &s_cos[j]);
  }
  if (a.bias != nullptr) {
#pragma unroll
    for (int i = 0; i < HPW; ++i) {
      const int h = warp + i * warps;
      if (h < n) {
        const float4 b = Four<float>::load(a.bias + h * ROPE_HD + d);
        v[i] = make_float4(v[i].x + b.x, v[i].y + b.y, v[i].z + b.z, v[i].w + b.w);
      }
    }
  }
  float ss[HPW];
  if (normed) {
#pragma unroll
    for (int i = 0; i < HPW; ++i) ss[i] = qb_warp_sum(squares(v[i]));
    if (a.norm_kind == NORM_PER_LAYER && lane == 0) {
#pragma unroll
      for (int i = 0; i < HPW; ++i) s_sum[warp + i * warps] = ss[i];
    }
  }
  __syncthreads();
  float rq = 1.f, rk = 1.f;
  if (a.norm_kind == NORM_PER_LAYER) {
    float tq = 0.f, tk = 0.f;
    for (int h = lane; h < nk; h += 32) {
      const float s = s_sum[h];
      tq += h < nq ? s : 0.f;
      tk += h < nq ? 0.f : s;
    }
    rq = rsqrtf(qb_warp_sum(tq) / (float)(nq * ROPE_HD) + a.eps);
    rk = rsqrtf(qb_warp_sum(tk) / (float)max(a.nkv * ROPE_HD, 1) + a.eps);
  }
  const float temp = a.temp_every > 0 ? 1.f + a.temp_coef * logf((float)((pos + 1) / a.temp_every) + 1.f) : 1.f;
  // this lane's pairs: cos and sin of pair j .. j + 3 (halves: the first turns by a c - b s, so its sines change sign), or of j and j + 1
  // (neighbours)
  const bool turns = d < a.rd, upper = d >= half;
  float4 c4 = make_float4(1.f, 1.f, 1.f, 1.f), s4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (turns) {
    if (a.interleaved) {
      c4.x = s_cos[d / 2]; c4.y = s_cos[d / 2 + 1];
      s4.x = s_sin[d / 2]; s4.y = s_sin[d / 2 + 1];
    } else {
      const int j = upper ? d - half : d;
      c4 = *reinterpret_cast<const float4*>(&s_cos[j]);
      s4 = *reinterpret_cast<const float4*>(&s_sin[j]);
      if (!upper) s4 = negated(s4);
    }
  }
  const int partner = turns && !a.interleaved ? (upper ? lane - half / 4 : lane + half / 4) : lane;
  const bool cache = writes && page >= 0 && page < a.num_pages;
  const int slot = a.page_shift >= 0 ? pos & (a.page_size - 1) : pos % a.page_size;
  const size_t at = ((size_t)(cache ? page : 0) * a.nkv * a.page_size + slot) * ROPE_HD + d;      // of kv head 0
  const int head_step = a.page_size * ROPE_HD;
  A* q_row = q_out + (size_t)t * nq * ROPE_HD + d;
#pragma unroll
  for (int i = 0; i < HPW; ++i) {
    const int h = warp + i * warps;          // the same for the whole warp
    if (h >= n) continue;
    const int hv = h - (a.tied_v ? nq : nk);
    if (cache && hv >= 0) {                  // values go out as they are (blended with an earlier layer's where asked)
      float4 x = v[i];
      const size_t own = ((size_t)t * a.nkv + hv) * ROPE_HD + d;
      if (a.v_export != nullptr) Four<float>::store(a.v_export + own, x);
      if (a.v_first != nullptr) {
        const float lam = a.v_lambda[0];
        const float4 f = Four<float>::load(a.v_first + own);
        x = make_float4((1.f - lam) * x.x + lam * f.x, (1.f - lam) * x.y + lam * f.y, (1.f - lam) * x.z + lam * f.z,
                        (1.f - lam) * x.w + lam * f.w);
      }
      Four<A>::store(v_cache + at + hv * head_step, x);
    }
    if (h >= nk) continue;
    float4 x = v[i];
    if (normed) {
      const float r = a.norm_kind == NORM_PER_LAYER ? (h < nq ? rq : rk) : rsqrtf(ss[i] / (float)ROPE_HD + a.eps);
      x = make_float4(x.x * r, x.y * r, x.z * r, x.w * r);
      if (gained) {
        const float4 g = EARLY ? w[EARLY ? i : 0] : gains(h);
        x = make_float4(g.x * x.x, g.y * x.y, g.z * x.z, g.w * x.w);
      }
    }
    if (a.interleaved) {
      if (turns) x = turned_pairs(x, c4.x, s4.x, c4.y, s4.y);
    } else if (half > 0) {
      const float4 o = make_float4(__shfl_sync(0xffffffffu, x.x, partner), __shfl_sync(0xffffffffu, x.y, partner),
                                   __shfl_sync(0xffffffffu, x.z, partner), __shfl_sync(0xffffffffu, x.w, partner));
      if (turns) x = turned(x, c4, o, s4);
    }
    if (h < nq) {
      if (a.temp_every > 0 || a.head_scale != nullptr) {
        const float m = a.head_scale != nullptr ? temp * a.head_scale[h] : temp;
        x = make_float4(x.x * m, x.y * m, x.z * m, x.w * m);
      }
      Four<A>::store(q_row + h * ROPE_HD, x);
    } else if (cache) {
      Four<A>::store(k_cache + at + (h - nq) * head_step, x);
    }
  }
  if (writes && !cache && threadIdx.x == 0) qb_set_status(a.status, QB_STATUS_BAD_PAGE, page, 2);
}

// ---------------------------------------------------------------------------------------------
// The same for many tokens, in about half the instructions: a half warp takes a head, a warp PPW pairs of heads, a lane the four elements
// of two lanes of the kernel above, d .. d + 3 and 64 + d .. 64 + d + 3.  The first of its exchanges is then an addition in the lane and the others
// leave each lane with one head's sum (the same additions in the same order, so that a token's numbers do not depend on the step);
// pairs meet by a shuffle among the first 64 elements or, where all 128 turn, in the lane.  Bound by instructions still (the bytes
// alone: 64 us for the 12,800 tokens below).  48 + 8 + 8 heads in bfloat16, 64 of 128 elements turned, a norm over all heads: 93 tokens 15.4 -> 12.3 us,
// 2,048 39.9 -> 31.7, 12,800 172 -> 126; 24 + 4 + 4, a norm a head, 12,800 tokens 99 -> 79; 16 + 4 + 4 from float32, neighbours, 59 -> 58.
// ---------------------------------------------------------------------------------------------
template <typename IN, typename A, int PPW>
__global__ void __launch_bounds__(512, 2)
qknorm_rope_pairs_kernel(const IN* qkv, A* __restrict__ q_out, A* __restrict__ k_cache, A* __restrict__ v_cache,
                         const RopeArgs a) {
  static_assert(PPW == 2 || PPW == 4, "one or two exchanges that halve a lane's sums");
  qb_follow();
  __shared__ __align__(16) float s_cos[ROPE_HD / 2], s_sin[ROPE_HD / 2];
  __shared__ float s_sum[ROPE_HD];
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, sub = lane & 15, side = lane >> 4;
  const int nq = a.nq, nk = nq + a.nkv, n = nk + (a.tied_v ? 0 : a.nkv), half = a.rd / 2, d = sub * 4;
  const bool writes = k_cache != nullptr, normed = a.norm_kind != NORM_NONE, gained = normed && a.q_norm_w != nullptr;
  const IN* row = qkv + (size_t)t * a.row_stride + d;
  int pos = 0, page = -1;                // asked for first: a chain of dependent loads
  if (writes || a.temp_every > 0) pos = a.tok_pos[t];
  auto head = [&](int i) { return 2 * (warp + i * warps) + side; };
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[PPW][2];
#pragma unroll
  for (int i = 0; i < PPW; ++i) {
    const int h = head(i);
#pragma unroll
    for (int e = 0; e < 2; ++e) v[i][e] = h < n ? Four<IN>::load(row + h * ROPE_HD + 64 * e) : none;
  }
  if (writes) {
    const int nth = a.page_shift >= 0 ? pos >> a.page_shift : pos / a.page_size;
    page = a.block_table[(size_t)a.tok_req[t] * a.bt_stride + nth];
  }
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    const int ax = a.pair_axis ? a.pair_axis[j] : 0;
    const float ang = (float)a.positions[(size_t)t * a.n_axes + ax] * a.inv_freq[j];
    sincosf(ang, &s_sin[j], &s_cos[j]);
  }
  if (a.bias != nullptr) {
#pragma unroll
    for (int i = 0; i < PPW; ++i) {
      const int h = head(i);
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (h < n) {
          const float4 b = Four<float>::load(a.bias + h * ROPE_HD + d + 64 * e);
          v[i][e] = make_float4(v[i][e].x + b.x, v[i][e].y + b.y, v[i][e].z + b.z, v[i][e].w + b.w);
        }
    }
  }
  float sum = 0.f;                       // of the pair `own` of this warp
  const int own = PPW == 4 ? (sub >> 2 & 3) : sub >> 3;
  if (normed) {
    float s[PPW];
#pragma unroll
    for (int i = 0; i < PPW; ++i) s[i] = squares(v[i][0]) + squares(v[i][1]);
#pragma unroll
    for (int x = 8, m = PPW; x > 0; x >>= 1) {
      if (m > 1) {
        m >>= 1;
        const bool up = sub & x;
#pragma unroll
        for (int i = 0; i < PPW / 2; ++i) {
          if (i >= m) break;
          const float give = up ? s[i] : s[i + m], keep = up ? s[i + m] : s[i];
          s[i] = keep + __shfl_xor_sync(0xffffffffu, give, x);
        }
      } else {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], x);
      }
    }
    sum = s[0];
    if (a.norm_kind == NORM_PER_LAYER && sub % (16 / PPW) == 0 && head(own) < n) s_sum[head(own)] = sum;
  }
  __syncthreads();
  float rq = 1.f, rk = 1.f;
  if (a.norm_kind == NORM_PER_LAYER) {
    float tq = 0.f, tk = 0.f;
    for (int h = lane; h < nk; h += 32) {
      const float s = s_sum[h];
      tq += h < nq ? s : 0.f;
      tk += h < nq ? 0.f : s;
    }
    rq = rsqrtf(qb_warp_sum(tq) / (float)(nq * ROPE_HD) + a.eps);
    rk = rsqrtf(qb_warp_sum(tk) / (float)max(a.nkv * ROPE_HD, 1) + a.eps);
  } else if (normed) {
    rq = rsqrtf(sum / (float)ROPE_HD + a.eps);      // of the pair `own`
  }
  const float temp = a.temp_every > 0 ? 1.f + a.temp_coef * logf((float)((pos + 1) / a.temp_every) + 1.f) : 1.f;
  // halves: cos and sin of pair j .. j + 3 (the first turns by a c - b s: within 64 elements its lane's sines change sign); neighbours: x, y of
  // the lane's first four elements, z, w of the others
  const bool turns = d < a.rd, turns2 = 64 + d < a.rd, upper = d >= half;
  float4 c4 = make_float4(1.f, 1.f, 1.f, 1.f), s4 = none;
  if (a.interleaved) {
    if (turns) { c4.x = s_cos[d / 2]; c4.y = s_cos[d / 2 + 1]; s4.x = s_sin[d / 2]; s4.y = s_sin[d / 2 + 1]; }
    if (turns2) { c4.z = s_cos[32 + d / 2]; c4.w = s_cos[33 + d / 2]; s4.z = s_sin[32 + d / 2]; s4.w = s_sin[33 + d / 2]; }
  } else if (turns) {
    const int j = upper ? d - half : d;
    c4 = *reinterpret_cast<const float4*>(&s_cos[j]);
    s4 = *reinterpret_cast<const float4*>(&s_sin[j]);
    if (!upper) s4 = negated(s4);
  }
  const int partner = turns ? (upper ? lane - half / 4 : lane + half / 4) : lane;      // (half at most 32)
  const bool cache = writes && page >= 0 && page < a.num_pages;
  const int slot = a.page_shift >= 0 ? pos & (a.page_size - 1) : pos % a.page_size;
  const size_t at = ((size_t)(cache ? page : 0) * a.nkv * a.page_size + slot) * ROPE_HD + d;      // of kv head 0
  const int head_step = a.page_size * ROPE_HD;
  A* q_row = q_out + (size_t)t * nq * ROPE_HD + d;
#pragma unroll
  for (int i = 0; i < PPW; ++i) {
    const int h = head(i), first = h - side;      // first: the same for the whole warp
    if (first >= n) continue;
    const int hv = h - (a.tied_v ? nq : nk);
    if (cache && hv >= 0 && h < n) {         // values go out as they are (blended with an earlier layer's where asked)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4 x = v[i][e];
        const size_t mine = ((size_t)t * a.nkv + hv) * ROPE_HD + d + 64 * e;
        if (a.v_export != nullptr) Four<float>::store(a.v_export + mine, x);
        if (a.v_first != nullptr) {
          const float lam = a.v_lambda[0];
          const float4 f = Four<float>::load(a.v_first + mine);
          x = make_float4((1.f - lam) * x.x + lam * f.x, (1.f - lam) * x.y + lam * f.y, (1.f - lam) * x.z + lam * f.z,
                          (1.f - lam) * x.w + lam * f.w);
        }
        Four<A>::store(v_cache + at + hv * head_step + 64 * e, x);
      }
    }
    if (first >= nk) continue;
    float4 x = v[i][0], y = v[i][1];
    if (normed) {
      float r = h < nq ? rq : rk;
      if (a.norm_kind == NORM_PER_HEAD) r = __shfl_sync(0xffffffffu, rq, side * 16 + i * (16 / PPW));
      x = make_float4(x.x * r, x.y * r, x.z * r, x.w * r);
      y = make_float4(y.x * r, y.y * r, y.z * r, y.w * r);
      if (gained && h < nk) {
        const float* w = (h < nq ? a.q_norm_w : a.k_norm_w) + (a.norm_kind == NORM_PER_LAYER ? (h < nq ? h : h - nq) * ROPE_HD : 0) + d;
        const float4 g = Four<float>::load(w), g2 = Four<float>::load(w + 64);
        x = make_float4(g.x * x.x, g.y * x.y, g.z * x.z, g.w * x.w);
        y = make_float4(g2.x * y.x, g2.y * y.y, g2.z * y.z, g2.w * y.w);
      }
    }
    if (a.interleaved) {
      if (turns) x = turned_pairs(x, c4.x, s4.x, c4.y, s4.y);
      if (turns2) y = turned_pairs(y, c4.z, s4.z, c4.w, s4.w);
    } else if (half == 64) {                   // s4 holds the first halves' signs
      const float4 o = x;
      x = turned(x, c4, y, s4);
      y = turned(y, c4, o, negated(s4));
    } else if (half > 0) {
      const float4 o = make_float4(__shfl_sync(0xffffffffu, x.x, partner), __shfl_sync(0xffffffffu, x.y, partner),
                                   __shfl_sync(0xffffffffu, x.z, partner), __shfl_sync(0xffffffffu, x.w, partner));
      if (turns) x = turned(x, c4, o, s4);
    }
    if (h < nq) {
      if (a.temp_every > 0 || a.head_scale != nullptr) {
        const float m = a.head_scale != nullptr ? temp * a.head_scale[h] : temp;
        x = make_float4(x.x * m, x.y * m, x.z * m, x.w * m);
        y = make_float4(y.x * m, y.y * m, y.z * m, y.w * m);
      }
      Four<A>::store(q_row + h * ROPE_HD, x);
      Four<A>::store(q_row + h * ROPE_HD + 64, y);
    } else if (cache && h < nk) {
      Four<A>::store(k_cache + at + (h - nq) * head_step, x);
      Four<A>::store(k_cache + at + (h - nq) * head_step + 64, y);
    }
  }
  if (writes && !cache && threadIdx.x == 0) qb_set_status(a.status, QB_STATUS_BAD_PAGE, page, 2);
}

template <typename IN, typename A>
static void qknorm_rope_heads(const void* qkv, void* q_out, void* k_cache, void* v_cache, const RopeArgs& a, int T, cudaStream_t stream) {
  const int heads = a.nq + a.nkv * (a.tied_v ? 1 : 2);
  if (T > 64 && (a.interleaved || a.rd <= 64 || a.rd == ROPE_HD)) {      // (pairs of other widths lie in two lanes' different halves)
    const int pairs = (heads + 1) / 2, ppw = heads <= 32 ? 2 : 4, threads = (pairs + ppw - 1) / ppw * 32;
    if (ppw == 2) qb_launch(qknorm_rope_pairs_kernel<IN, A, 2>, T, threads, 0, stream, (const IN*)qkv, (A*)q_out, (A*)k_cache, (A*)v_cache, a);
    else qb_launch(qknorm_rope_pairs_kernel<IN, A, 4>, T, threads, 0, stream, (const IN*)qkv, (A*)q_out, (A*)k_cache, (A*)v_cache, a);
    return;
  }
  // few tokens: two heads a warp, so that a token is one short wait; many: four or eight loads in flight a lane
  const int hpw = T <= 64 && heads <= 64 ? 2 : heads <= 32 ? 4 : 8;
  const int threads = (heads + hpw - 1) / hpw * 32;
#define QB_HEADS(N) \
  qb_launch(qknorm_rope_heads_kernel<IN, A, N>, T, threads, 0, stream, (const IN*)qkv, (A*)q_out, (A*)k_cache, (A*)v_cache, a)
  if (hpw == 2) QB_HEADS(2);
  else if (hpw == 4) QB_HEADS(4);
  else QB_HEADS(8);
#undef QB_HEADS
}

extern "C" int qb_qknorm_rope_write(
    const void* qkv, int in_dtype, int dtype, int row_stride, void* q_out, void* k_cache, void* v_cache, const float* q_norm_w,
    const float* k_norm_w, int norm_kind, float eps, const float* inv_freq, const int* pair_axis,
    const int* positions, int n_axes, const int* tok_pos, const int* tok_req, const int* block_table,
    int bt_stride, int T, int nq, int nkv, int hd, int vd, int has_kv, int tied_v, int rd, int interleaved, float temp_coef,
    int temp_every, int page_size, int num_pages, const float* bias, const float* v_first, const float* v_lambda, float* v_export,
    const float* head_scale, int* status, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (rd % 2 || rd > hd || rd < 0 || nq <= 0 || nkv <= 0 || page_size <= 0 || hd <= 0 || vd <= 0) return QB_ERR_BAD_ARG;
  // a norm over the whole row needs gains; a per-head norm may have none (both null)
  if (norm_kind == NORM_PER_LAYER && (q_norm_w == nullptr || (has_kv && k_norm_w == nullptr))) return QB_ERR_BAD_ARG;
  if (norm_kind == NORM_PER_HEAD && q_norm_w != nullptr && has_kv && k_norm_w == nullptr) return QB_ERR_BAD_ARG;
  if (norm_kind == NORM_PER_HEAD && q_norm_w == nullptr && k_norm_w != nullptr) return QB_ERR_BAD_ARG;
  if ((v_first != nullptr && v_lambda == nullptr) || ((v_first != nullptr || v_export != nullptr) && !has_kv)) return QB_ERR_BAD_ARG;
  if (in_dtype != dtype && in_dtype != QB_F32) return QB_ERR_BAD_ARG;
  if (!has_kv && k_cache != nullptr) return QB_ERR_BAD_ARG;
  const int nk = has_kv ? nkv : 0;
  if (tied_v && (vd != hd || !has_kv)) return QB_ERR_BAD_ARG;
  if (row_stride < nq * hd + nk * (hd + (tied_v ? 0 : vd))) return QB_ERR_BAD_ARG;
  // rows are moved in 16-byte pieces where every piece starts on such a boundary; else element by element
  const int vec = (hd % 8 == 0 && vd % 8 == 0 && row_stride % 8 == 0 && ((uintptr_t)qkv & 15) == 0) ? 1 : 0;
  // heads of 128, pairs that fall on whole lanes, every address on a lane's piece; at most 16 warps of eight heads
  const uintptr_t all = (uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)q_norm_w | (uintptr_t)k_norm_w |
                        (uintptr_t)bias | (uintptr_t)v_first | (uintptr_t)v_export;
  if (vec && hd == ROPE_HD && vd == ROPE_HD && (interleaved ? rd % 4 : rd % 8) == 0 && (all & 15) == 0 &&
      nq + nk * (tied_v ? 1 : 2) <= 128) {
    int shift = -1;
    for (int i = 0; i < 31; ++i)
      if (page_size == 1 << i) shift = i;
    const RopeArgs a{row_stride, norm_kind, n_axes, bt_stride, nq, nk, tied_v, rd, interleaved, temp_every, page_size, shift, num_pages,
                     eps, temp_coef, q_norm_w, k_norm_w, inv_freq, bias, v_first, v_lambda, head_scale,
                     pair_axis, positions, tok_pos, tok_req, block_table, v_export, status};
    if (dtype == QB_F32) qknorm_rope_heads<float, float>(qkv, q_out, k_cache, v_cache, a, T, stream);
    else if (dtype == QB_BF16 && in_dtype == QB_F32) qknorm_rope_heads<float, __nv_bfloat16>(qkv, q_out, k_cache, v_cache, a, T, stream);
    else if (dtype == QB_BF16) qknorm_rope_heads<__nv_bfloat16, __nv_bfloat16>(qkv, q_out, k_cache, v_cache, a, T, stream);
    else return QB_ERR_BAD_ARG;
    QB_LAUNCH_CHECK();
    return 0;
  }
  const size_t smem = (size_t)((nq + nk) * hd + rd + 32 + nq + nk) * sizeof(float);
  if (smem > 200 * 1024) return QB_ERR_UNSUPPORTED;
#define QB_ROPE_LAUNCH(IN, A)                                                                                   \
  do {                                                                                                          \
    auto kern = qknorm_rope_write_kernel<IN, A>;                                                                \
    if (smem > 48 * 1024) {                                                                                     \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
      if (e != cudaSuccess) return (int)e;                                                                      \
    }                                                                                                           \
    kern<<<T, threads, smem, stream>>>((const IN*)qkv, row_stride, (A*)q_out, (A*)k_cache, (A*)v_cache, q_norm_w, \
                                       k_norm_w, norm_kind, eps, inv_freq, pair_axis, positions, n_axes, tok_pos, \
                                       tok_req, block_table, bt_stride, T, nq, nkv, hd, vd, has_kv, tied_v, rd,  \
                                       interleaved, temp_coef, temp_every, page_size, num_pages, vec, bias, v_first, v_lambda, v_export,  \
                                       head_scale, status);                                                              \
  } while (0)
  // steps of few tokens: more threads a token, so that each of the kernel's phases is short
  const int threads = T <= 64 ? 1024 : 256;
  if (dtype == QB_F32) QB_ROPE_LAUNCH(float, float);
  else if (dtype == QB_BF16 && in_dtype == QB_F32) QB_ROPE_LAUNCH(float, __nv_bfloat16);
  else if (dtype == QB_BF16) QB_ROPE_LAUNCH(__nv_bfloat16, __nv_bfloat16);
  else return QB_ERR_BAD_ARG;
#undef QB_ROPE_LAUNCH
  QB_LAUNCH_CHECK();
  return 0;
}
