// Paged causal attention over the cache, plain SIMT version (float32 arithmetic throughout).
//
// This is the kernel of the true 32-bit path, and the reference the tensor-core kernels are checked
// against.  Every token of the step is its own problem: token t of request r at absolute position p
// attends the keys [lo, p] of r's pages (lo = 0, or p-window+1 for a windowed layer), whatever else is
// in the batch, so prompt portions and single decoded tokens run in one launch.  K and V of the
// step's own tokens have been written to the pages before this kernel runs.
//
//   s = (q . k) * scale;  softmax over keys in float32;  out = P V
//   (src/quanta/minimax/attention.py:194-203; grouped heads: q head h reads kv head h / (nq/nkv))
// Keys (and queries) have `hd` elements a head, values and outputs `vd`; any positive sizes up to 256 (rows
// whose size is no multiple of the 16-byte vector are read element by element).
//
// Two kernels.  Head sizes that are multiples of 4: a block per (token, kv head, up to four of its q heads), the warps share the
// keys.  Other sizes: one warp per (token, q head): lanes own keys for the scores, then own dims for P V.
#include "rows_f32.cuh"

template <typename A> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float* o) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void load(const __nv_bfloat16* p, float* o) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};

constexpr int ATT_WARPS = 4;
constexpr int ATT_MAX_HD = 256;

template <typename A>
__global__ void paged_attention_simt_kernel(
    const A* __restrict__ q, const A* __restrict__ k_cache, const A* __restrict__ v_cache,
    A* __restrict__ out, const int* __restrict__ tok_pos, const int* __restrict__ tok_req,
    const int* __restrict__ block_table, int bt_stride, int T, int nq, int nkv, int hd, int vd, int page_size,
    int num_pages, float scale, int window, int vec, int* status) {
  extern __shared__ float qs_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long wid = (long)blockIdx.x * ATT_WARPS + warp;
  if (wid >= (long)T * nq) return;
  const int t = (int)(wid / nq), h = (int)(wid % nq);
  const int kvh = h / (nq / nkv);
  float* qs = qs_all + warp * hd;
  const A* qrow = q + ((size_t)t * nq + h) * hd;
  for (int d = lane; d < hd; d += 32) qs[d] = qb_to_float<A>(qrow[d]);
  __syncwarp();

  const int pos = tok_pos[t];
  const int* bt = block_table + (size_t)tok_req[t] * bt_stride;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;

  float m = -INFINITY, l = 0.f;
  float acc[ATT_MAX_HD / 32];
#pragma unroll
  for (int i = 0; i < ATT_MAX_HD / 32; ++i) acc[i] = 0.f;

  for (int kb = lo - (lo & 31); kb <= pos; kb += 32) {
    const int key = kb + lane;
    const bool valid = key >= lo && key <= pos;
    float s = -INFINITY;
    long base = -1;     // index of this lane's key row among all (page, kv head, slot) rows, in K and in V
    if (valid) {
      const int page = bt[key / page_size];
      if (page < 0 || page >= num_pages) {
        qb_set_status(status, QB_STATUS_BAD_PAGE, page, 3);
      } else {
        base = ((long)page * nkv + kvh) * page_size + key % page_size;
        const A* kp = k_cache + base * hd;
        float dot = 0.f;
        if (vec) {
          for (int d = 0; d < hd; d += Vec16<A>::N) {
            float kv[Vec16<A>::N];
            Vec16<A>::load(kp + d, kv);
#pragma unroll
            for (int i = 0; i < Vec16<A>::N; ++i) dot += qs[d + i] * kv[i];
          }
        } else {
          for (int d = 0; d < hd; ++d) dot += qs[d] * qb_to_float<A>(kp[d]);
        }
        s = dot * scale;
      }
    }
    const float mb = qb_warp_max(s);
    if (mb == -INFINITY) continue;
    const float m_new = fmaxf(m, mb);
    const float p = (base >= 0) ? expf(s - m_new) : 0.f;
    const float corr = expf(m - m_new);
    l = l * corr + qb_warp_sum(p);
#pragma unroll
    for (int i = 0; i < ATT_MAX_HD / 32; ++i) acc[i] *= corr;
    const int n_here = min(32, pos - kb + 1);
    for (int j = 0; j < n_here; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
      const long bj = __shfl_sync(0xffffffffu, base, j);
      if (bj < 0) continue;
      const A* vp = v_cache + bj * vd;
#pragma unroll
      for (int i = 0; i < ATT_MAX_HD / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < vd) acc[i] += pj * qb_to_float<A>(vp[d]);
      }
    }
    m = m_new;
  }
  A* orow = out + ((size_t)t * nq + h) * vd;
  const float inv_l = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int i = 0; i < ATT_MAX_HD / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < vd) orow[d] = qb_from_float<A>(acc[i] * inv_l);
  }
}

// ---------------------------------------------------------------------------------------------
// Head sizes that are multiples of 4.  A warp takes eight keys at a time: a key (and a value) row is one coalesced read of the
// warp, 16 bytes a lane (8 of bfloat16), all sixteen rows asked for at once and read once for GH q heads; the 8 x GH scores are
// summed over the lanes together (rows_f32.cuh), so that lane 4 j + .. holds key j.  The eight warps of a block take turns of eight
// keys and their results are joined through shared memory in warp order.  Bound by the chain of a turn when there are few tokens:
// the float32 steps of 4 requests of some 130 tokens and their prompts took 145 us a launch on average with a warp a (token, head) and
// a key a lane, 11 us with this.
// ---------------------------------------------------------------------------------------------
template <typename A> struct Vec4;
template <> struct Vec4<float> {
  __device__ static __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
  __device__ static __forceinline__ void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};
template <> struct Vec4<__nv_bfloat16> {
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

constexpr int ATS_WARPS = 8, ATS_KEYS = 8;

// GH q heads a block (1, 2 or 4); NV groups of 128 elements a row at most.
template <typename A, int GH, int NV>
__global__ void __launch_bounds__(ATS_WARPS * 32)
paged_attention_rows_kernel(const A* __restrict__ q, const A* __restrict__ k_cache, const A* __restrict__ v_cache, A* __restrict__ out,
                            const int* __restrict__ tok_pos, const int* __restrict__ tok_req, const int* __restrict__ block_table,
                            int bt_stride, int nq, int nkv, int hd, int vd, int page_size, int num_pages, float scale, int window,
                            int* status) {
  extern __shared__ __align__(16) float ats_acc[];           // [warps][GH][vd]
  __shared__ float s_m[ATS_WARPS][GH], s_l[ATS_WARPS][GH];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int heads_of_kv = nq / nkv, chunks = heads_of_kv / GH;
  const int t = blockIdx.x / (nkv * chunks), rest = blockIdx.x % (nkv * chunks);
  const int kvh = rest / chunks, h0 = kvh * heads_of_kv + (rest % chunks) * GH;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);

  float4 qv[GH][NV], acc[GH][NV];
#pragma unroll
  for (int g = 0; g < GH; ++g)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int d = lane * 4 + 128 * i;
      qv[g][i] = d < hd ? Vec4<A>::load(q + ((size_t)t * nq + h0 + g) * hd + d) : zero;
      acc[g][i] = zero;
    }
  const int pos = tok_pos[t];
  const int* bt = block_table + (size_t)tok_req[t] * bt_stride;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  float m = -INFINITY, l = 0.f;                              // of this lane's head, (lane & 3) / (4 / GH)
  for (int kb = lo + warp * ATS_KEYS; kb <= pos; kb += ATS_WARPS * ATS_KEYS) {
    long base = -1;        // lane j < 8: index of key kb + j's row among all (page, kv head, slot) rows, in K and in V
    if (lane < ATS_KEYS && kb + lane <= pos) {
      const int key = kb + lane, page = bt[key / page_size];
      if (page < 0 || page >= num_pages) qb_set_status(status, QB_STATUS_BAD_PAGE, page, 3);
      else base = ((long)page * nkv + kvh) * page_size + key % page_size;
    }
    float4 kv[ATS_KEYS][NV], vv[ATS_KEYS][NV];
#pragma unroll
    for (int j = 0; j < ATS_KEYS; ++j) {
      const long bj = __shfl_sync(0xffffffffu, base, j);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int d = lane * 4 + 128 * i;
        kv[j][i] = bj >= 0 && d < hd ? Vec4<A>::load(k_cache + bj * hd + d) : zero;
        vv[j][i] = bj >= 0 && d < vd ? Vec4<A>::load(v_cache + bj * vd + d) : zero;
      }
    }
    float s[ATS_KEYS * GH];
#pragma unroll
    for (int j = 0; j < ATS_KEYS; ++j)
#pragma unroll
      for (int g = 0; g < GH; ++g) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          dot = fmaf(qv[g][i].x, kv[j][i].x, dot);
          dot = fmaf(qv[g][i].y, kv[j][i].y, dot);
          dot = fmaf(qv[g][i].z, kv[j][i].z, dot);
          dot = fmaf(qv[g][i].w, kv[j][i].w, dot);
        }
        s[j * GH + g] = dot;
      }
    qb_sum_values<ATS_KEYS * GH>(s, lane);                   // lane: key lane / 4, head (lane & 3) / (4 / GH)
    const bool seen = __shfl_sync(0xffffffffu, base, lane >> 2) >= 0;
    const float mine = seen ? s[0] * scale : -INFINITY;
    float top = mine;
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    const float m_new = fmaxf(m, top);
    const float p = seen ? expf(mine - m_new) : 0.f;
    const float corr = m_new > -INFINITY ? expf(m - m_new) : 1.f;
    float sum = p;
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    l = l * corr + sum;
    m = m_new;
#pragma unroll
    for (int g = 0; g < GH; ++g) {
      const float c = __shfl_sync(0xffffffffu, corr, g * (4 / GH));
#pragma unroll
      for (int i = 0; i < NV; ++i) acc[g][i] = make_float4(acc[g][i].x * c, acc[g][i].y * c, acc[g][i].z * c, acc[g][i].w * c);
#pragma unroll
      for (int j = 0; j < ATS_KEYS; ++j) {
        const float pj = __shfl_sync(0xffffffffu, p, 4 * j + g * (4 / GH));
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          acc[g][i].x = fmaf(pj, vv[j][i].x, acc[g][i].x);
          acc[g][i].y = fmaf(pj, vv[j][i].y, acc[g][i].y);
          acc[g][i].z = fmaf(pj, vv[j][i].z, acc[g][i].z);
          acc[g][i].w = fmaf(pj, vv[j][i].w, acc[g][i].w);
        }
      }
    }
  }
  if (lane < 4 && lane % (4 / GH) == 0) {
    s_m[warp][lane / (4 / GH)] = m;
    s_l[warp][lane / (4 / GH)] = l;
  }
#pragma unroll
  for (int g = 0; g < GH; ++g)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int d = lane * 4 + 128 * i;
      if (d < vd) *reinterpret_cast<float4*>(ats_acc + ((size_t)warp * GH + g) * vd + d) = acc[g][i];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < GH * vd / 4; i += ATS_WARPS * 32) {
    const int g = i / (vd / 4), d = (i % (vd / 4)) * 4;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATS_WARPS; ++w) top = fmaxf(top, s_m[w][g]);
    float sum = 0.f;
    float4 o = zero;
#pragma unroll
    for (int w = 0; w < ATS_WARPS; ++w) {
      const float f = s_m[w][g] > -INFINITY ? expf(s_m[w][g] - top) : 0.f;
      const float4 a = *reinterpret_cast<const float4*>(ats_acc + ((size_t)w * GH + g) * vd + d);
      sum = fmaf(s_l[w][g], f, sum);
      o = make_float4(fmaf(a.x, f, o.x), fmaf(a.y, f, o.y), fmaf(a.z, f, o.z), fmaf(a.w, f, o.w));
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    Vec4<A>::store(out + ((size_t)t * nq + h0 + g) * vd + d, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
  }
}

template <typename A, int GH>
static void paged_attention_rows(int NV, int blocks, const A* q, const A* k, const A* v, A* out, const int* tok_pos, const int* tok_req,
                                 const int* bt, int bt_stride, int nq, int nkv, int hd, int vd, int page_size, int num_pages, float scale,
                                 int window, int* status, cudaStream_t stream) {
  const size_t smem = (size_t)ATS_WARPS * GH * vd * sizeof(float);            // at most 32 KB
  if (NV == 1)
    paged_attention_rows_kernel<A, GH, 1><<<blocks, ATS_WARPS * 32, smem, stream>>>(q, k, v, out, tok_pos, tok_req, bt, bt_stride, nq,
                                                                                   nkv, hd, vd, page_size, num_pages, scale, window, status);
  else
    paged_attention_rows_kernel<A, GH, 2><<<blocks, ATS_WARPS * 32, smem, stream>>>(q, k, v, out, tok_pos, tok_req, bt, bt_stride, nq,
                                                                                   nkv, hd, vd, page_size, num_pages, scale, window, status);
}

extern "C" int qb_paged_attention_simt(const void* q, int dtype, const void* k_cache, const void* v_cache,
                                       void* out, const int* tok_pos, const int* tok_req,
                                       const int* block_table, int bt_stride, int T, int nq, int nkv, int hd,
                                       int vd, int page_size, int num_pages, float scale, int window, int* status,
                                       cudaStream_t stream) {
  if (T <= 0) return 0;
  if (hd <= 0 || vd <= 0 || hd > ATT_MAX_HD || vd > ATT_MAX_HD || nq % nkv || page_size <= 0) return QB_ERR_UNSUPPORTED;
  const uintptr_t all = (uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out;
  if (hd % 4 == 0 && vd % 4 == 0 && (all & 15) == 0) {
    const int per_kv = nq / nkv, GH = per_kv % 4 == 0 ? 4 : per_kv % 2 == 0 ? 2 : 1, NV = hd > 128 || vd > 128 ? 2 : 1;
    const long blocks_l = (long)T * nq / GH;
    if (blocks_l > 0x7fffffffL) return QB_ERR_UNSUPPORTED;
#define QB_ATS(G)                                                                                                                  \
  paged_attention_rows<A, G>(NV, (int)blocks_l, (const A*)q, (const A*)k_cache, (const A*)v_cache, (A*)out, tok_pos, tok_req,       \
                             block_table, bt_stride, nq, nkv, hd, vd, page_size, num_pages, scale, window, status, stream)
    QB_DISPATCH_DTYPE(dtype, A, {
      if (GH == 4) QB_ATS(4);
      else if (GH == 2) QB_ATS(2);
      else QB_ATS(1);
    });
#undef QB_ATS
    QB_LAUNCH_CHECK();
    return 0;
  }
  const int vec = (hd % 8 == 0 && ((uintptr_t)k_cache & 15) == 0) ? 1 : 0;      // key rows start on 16 bytes
  const long warps = (long)T * nq;
  const int blocks = (int)((warps + ATT_WARPS - 1) / ATT_WARPS);
  const size_t smem = (size_t)ATT_WARPS * hd * sizeof(float);
  QB_DISPATCH_DTYPE(dtype, A,
                    paged_attention_simt_kernel<A><<<blocks, ATT_WARPS * 32, smem, stream>>>(
                        (const A*)q, (const A*)k_cache, (const A*)v_cache, (A*)out, tok_pos, tok_req,
                        block_table, bt_stride, T, nq, nkv, hd, vd, page_size, num_pages, scale, window, vec, status));
  QB_LAUNCH_CHECK();
  return 0;
}
