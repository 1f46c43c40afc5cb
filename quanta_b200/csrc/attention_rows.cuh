// Paged attention of few queries, float32 arithmetic, head sizes that are multiples of 4 up to 256: a block per (token, kv head, up to
// four of its q heads, range of its keys).
//
// A warp takes eight keys at a time: a key (and a value) row is one coalesced read of the warp, 16 bytes a lane (8 of
// bfloat16), all sixteen rows asked for at once and read once for GH q heads; the 8 x GH scores are summed over the lanes together
// (rows_f32.cuh), so that lane 4 j + .. holds key j and applies cap and bias to it once.  The eight warps of a block take turns of
// eight keys and their results are joined through shared memory in warp order; with n_split > 1 a block takes one of that many ranges of the
// keys and leaves (max, sum, sums of values) for a second launch.  Bound by the chain of a turn (2.6 us: a look-up, a read of
// memory, the sums) when there are few tokens: the float32 steps of 4 requests of some 130 tokens and their prompts took 145 us a launch with a warp a
// (token, head) and a key a lane, 11 us with this; with a window of 1,024, 16 + 4 heads in float32 with biases by distance, ranges of 256 keys: 16
// tokens 42 us with a warp a range, 25 with this (joined in both), a prompt of 300 tokens 102 and 58, of 1,500 1,176 and 828.
#pragma once
#include "rows_f32.cuh"

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

struct RowsAttention {
  const int *tok_pos, *tok_req, *block_table;
  int bt_stride, T, nq, nkv, hd, vd, page_size, num_pages;
  float scale, cap;              // cap > 0: score <- cap tanh(score / cap)
  int window, chunk;             // > 0: the last `window` keys; the keys of the token's own chunk of positions
  const float* dist_bias;        // [window, nq] by distance, or null
  const float* sink;             // [nq], or null
  int n_split;                   // ranges of a token's keys
  float* part;                   // n_split > 1: [T, nq, n_split, 2 + vd]
  int* status;
};

// GH q heads a block (1, 2 or 4); NV groups of 128 elements a row at most.
template <typename A, int GH, int NV>
__global__ void __launch_bounds__(ATS_WARPS * 32)
paged_attention_rows_kernel(const A* __restrict__ q, const A* __restrict__ k_cache, const A* __restrict__ v_cache, A* __restrict__ out,
                            const RowsAttention P) {
  extern __shared__ __align__(16) float ats_acc[];           // [warps][GH][vd]
  __shared__ float s_m[ATS_WARPS][GH], s_l[ATS_WARPS][GH];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nq = P.nq, nkv = P.nkv, hd = P.hd, vd = P.vd, page_size = P.page_size;
  const int heads_of_kv = nq / nkv, chunks = heads_of_kv / GH;
  const int unit = blockIdx.x / P.n_split, split = blockIdx.x % P.n_split;
  const int t = unit / (nkv * chunks), rest = unit % (nkv * chunks);
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
  const int pos = P.tok_pos[t];
  const int* bt = P.block_table + (size_t)P.tok_req[t] * P.bt_stride;
  int lo = P.window > 0 && pos - P.window + 1 > 0 ? pos - P.window + 1 : 0, end = pos;
  if (P.chunk > 0) lo = max(lo, pos / P.chunk * P.chunk);
  if (P.n_split > 1) {           // this block's range, whole turns of its warps
    const int per = ((pos - lo + P.n_split) / P.n_split + ATS_WARPS * ATS_KEYS - 1) / (ATS_WARPS * ATS_KEYS) * (ATS_WARPS * ATS_KEYS);
    lo += split * per;
    end = min(pos, lo + per - 1);
  }
  const int my_head = h0 + (lane & 3) / (4 / GH);
  float m = -INFINITY, l = 0.f;                              // of this lane's head, (lane & 3) / (4 / GH)
  for (int kb = lo + warp * ATS_KEYS; kb <= end; kb += ATS_WARPS * ATS_KEYS) {
    long base = -1;        // lane j < 8: index of key kb + j's row among all (page, kv head, slot) rows, in K and in V
    if (lane < ATS_KEYS && kb + lane <= end) {
      const int key = kb + lane, page = bt[key / page_size];
      if (page < 0 || page >= P.num_pages) qb_set_status(P.status, QB_STATUS_BAD_PAGE, page, 3);
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
    float mine = s[0] * P.scale;
    if (P.cap > 0.f) mine = P.cap * tanhf(mine / P.cap);
    if (P.dist_bias != nullptr && seen) mine += P.dist_bias[(size_t)(pos - kb - (lane >> 2)) * nq + my_head];
    if (!seen) mine = -INFINITY;
    float top = mine;
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    // keys may have scores of minus infinity (a bias that masks them): while nothing else has been seen, exponents are taken against 0
    const float m_new = fmaxf(m, top), ref = m_new > -INFINITY ? m_new : 0.f;
    const float p = seen ? expf(mine - ref) : 0.f;
    const float corr = expf(m - ref);
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
    if (P.n_split > 1) {
      float* prow = P.part + (((size_t)t * nq + h0 + g) * P.n_split + split) * (2 + (size_t)vd);
      if (d == 0) { prow[0] = top; prow[1] = sum; }
      prow[2 + d] = o.x; prow[3 + d] = o.y; prow[4 + d] = o.z; prow[5 + d] = o.w;
      continue;
    }
    if (P.sink != nullptr) {                    // one more score, whose value is zero
      const float sk = P.sink[h0 + g];
      if (sk > top) {
        const float f = top > -INFINITY ? expf(top - sk) : 0.f;
        sum *= f;
        o = make_float4(o.x * f, o.y * f, o.z * f, o.w * f);
        top = sk;
      }
      sum += expf(sk - top);
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    Vec4<A>::store(out + ((size_t)t * nq + h0 + g) * vd + d, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
  }
}

// Whether the kernel takes these sizes and addresses.
static bool rows_attention_takes(int nq, int nkv, int hd, int vd, const void* q, const void* k, const void* v, const void* out) {
  return hd > 0 && vd > 0 && hd <= 256 && vd <= 256 && nkv > 0 && nq % nkv == 0 && hd % 4 == 0 && vd % 4 == 0 &&
         (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) == 0;
}

// q heads a block of the kernel.
static int rows_attention_heads(int nq, int nkv) {
  const int per_kv = nq / nkv;
  return per_kv % 4 == 0 ? 4 : per_kv % 2 == 0 ? 2 : 1;
}

// Whether the kernel is faster than the one that gives a range of a token's keys to a warp for all q heads of a kv head.  A turn of 64 keys takes
// a block 2.6 us whatever the head size and the number of its q heads, so few blocks are always faster here, many where the rows are
// long and shared.  Measured on a B200 (ranges of the keys / here, us): 16 + 4 heads of 128, bfloat16, windows of 512, 16 tokens 25 / 17, 1,000 406 / 282;
// 8 + 8 of 64, 16 tokens 20 / 19, 1,000 301 / 459; 6 + 2 of 128, 64 tokens 1.4 times slower here; 16 + 4 of 16, float32, 1,000 tokens 154 / 303;
// 12 + 2 of 256, 64 tokens 142 / 249; 8 + 2 of 80, float32, 64 tokens 1.4 times slower, bfloat16 0.8.
static bool rows_attention_wins(bool f32, int T, int nq, int nkv, int hd) {
  const int GH = rows_attention_heads(nq, nkv);
  const long blocks = (long)T * nq / GH;
  if (blocks <= 64) return true;
  if (f32) return (GH == 4 && hd >= 64 && hd < 80 && blocks <= 1024) || (hd >= 112 && (GH > 1 || nq == nkv) && (hd <= 128 || GH == 4));
  return GH == 4 && (hd >= 80 || (hd >= 64 && blocks <= 256));
}

template <typename A>
static int rows_attention(const A* q, const A* k, const A* v, A* out, const RowsAttention& P, cudaStream_t stream) {
  const int GH = rows_attention_heads(P.nq, P.nkv), NV = P.hd > 128 || P.vd > 128 ? 2 : 1;
  const long blocks = (long)P.T * P.nq / GH * P.n_split;
  if (blocks > 0x7fffffffL) return QB_ERR_UNSUPPORTED;
  const size_t smem = (size_t)ATS_WARPS * GH * P.vd * sizeof(float);            // at most 32 KB
#define QB_ATS(G, N) paged_attention_rows_kernel<A, G, N><<<(int)blocks, ATS_WARPS * 32, smem, stream>>>(q, k, v, out, P)
#define QB_ATS_G(N)                 \
  do {                              \
    if (GH == 4) QB_ATS(4, N);      \
    else if (GH == 2) QB_ATS(2, N); \
    else QB_ATS(1, N);              \
  } while (0)
  if (NV == 1) QB_ATS_G(1);
  else QB_ATS_G(2);
#undef QB_ATS_G
#undef QB_ATS
  QB_LAUNCH_CHECK();
  return 0;
}
