// Attention of single tokens over the paged cache for heads of 128 and at most eight q heads a kv head (bfloat16, mma.sync).
//
//   out[t, h] = softmax_j(q[t, h] . k_j * scale) v_j       over the keys [lo, pos] of the token's request
//   (src/quanta/minimax/attention.py:194-203; float32 scores and sums, weights rounded to bfloat16 before P V, or with SPLIT as they
//   are: three bfloat16 parts hold a float32's 24 bits, three products a tile; a cap on the scores and a chunk of the sequence
//   besides the window)
//
// A warp works by itself, 16 keys at a time, until the end: its keys and values come by asynchronous copies of its own into a ring of
// three rounds, so it waits for no other warp, and the tensor cores take their operands as the rows lie.
//   S = Q K^T   (m16n8k16: rows are q heads, eight of them used; columns are keys).  The order of the inner dimension is free as long
//               as Q and K agree, so lane (g, t) takes the 16-byte pieces t, t + 4, t + 8, t + 12 of row g of Q and of K as four
//               fragments' worth: one 16-byte read each.
//   O^T += V^T P^T  (m16n8k16: rows are dims, columns q heads, the inner dimension the 16 keys).  P^T's fragment is what S's
//               accumulators hold; lane (g, t) reads pieces g and g + 8 of the rows 2t, 2t + 1, 2t + 8, 2t + 9 of V and pairs the
//               keys with byte permutations; row g of tile e is dim 8 g + e, row g + 8 is dim 64 + 8 g + e.
// Pieces are stored at p ^ 4 (row & 1) (K) and p ^ 2 (row / 2 & 3) (V), so that the eight lanes of a phase meet no bank twice.  Two rounds are
// on their way while one is used, their places in the cache looked up one round before: 16 KB a warp, 128 KB an SM (loads into registers,
// one round ahead, waited for the newest load with the oldest: 64 tokens of 1,600 keys on average 111 us, 91 us with this).  A unit is a (token,
// kv head); its keys go round the warps of a block and of the S blocks of a cluster, whose results are joined through (distributed)
// shared memory in a fixed order: one launch, no scratch in memory.
//
// Bound by the bytes of keys and values for many keys and by three memory latencies for few.  Measured on a B200, 48 + 8 heads, beside the
// persistent kernel of attention_mma.cu with its merge launch: see the rule in qb_attn_decode_direct_wins.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int DD_HD = 128, DD_KEYS = 16, DD_LD = DD_HD + 8, DD_MAX_WARPS = 8, DD_STAGES = 3;
constexpr int DD_ROUND = 2 * DD_KEYS * DD_HD;       // elements of a round: 16 rows of K, 16 of V

__device__ __forceinline__ void dd_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dd_copy16(uint32_t dst, const __nv_bfloat16* src, bool there) {      // zeros where it is not
  const int n = there ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float dd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t dd_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void dd_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float dd_remote(const float* p, int rank) {     // the same place in another block of the cluster
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t r;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
  return v;
}

struct DecodeArgs {
  const int *dec_tok, *tok_pos, *tok_req, *block_table;
  int bt_stride, nq, nkv, page_size, page_shift, num_pages, window, chunk, S, early;
  float scale, cap;
  int* status;
};

template <bool SPLIT>
__global__ void __launch_bounds__(DD_MAX_WARPS * 32)
attn_decode_direct_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k_cache,      // q: see qb_follow
                          const __nv_bfloat16* v_cache, __nv_bfloat16* __restrict__ out, const DecodeArgs P) {
  if (!P.early) qb_follow();
  extern __shared__ __align__(128) unsigned char dd_smem[];
  // rings first; then a warp's sums, a head's 128 numbers in the order 8 e + g | 64 + 8 e + g
  __nv_bfloat16* ring = reinterpret_cast<__nv_bfloat16*>(dd_smem);
  float (*s_o)[8][DD_LD] = reinterpret_cast<float (*)[8][DD_LD]>(dd_smem);
  __shared__ float s_m[DD_MAX_WARPS][8], s_l[DD_MAX_WARPS][8];
  __shared__ float s_po[8][DD_LD], s_pm[8], s_pl[8]; // the block's
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int unit = blockIdx.x / P.S, rank = blockIdx.x % P.S;
  const int tok = P.dec_tok[unit / P.nkv], kvh = unit % P.nkv, G = P.nq / P.nkv;
  const int pos = P.tok_pos[tok];
  int lo = P.window > 0 && pos - P.window + 1 > 0 ? pos - P.window + 1 : 0;
  if (P.chunk > 0) lo = max(lo, pos / P.chunk * P.chunk);
  constexpr float LOG2E = 1.4426950408889634f;
  const float scale_log2 = P.scale * LOG2E;
  const int* bt = P.block_table + (size_t)P.tok_req[tok] * P.bt_stride;

  // rounds of 16 keys: first, first + step, ... up to the group of the last key
  const int step = warps * P.S, last = pos / DD_KEYS;
  // lane l < 16: the row of key 16 r + l in K and V (of this kv head), -1 for keys that are not read
  auto place = [&](int r) -> int {
    const int key = r * DD_KEYS + (lane & 15);
    if (r > last || key < lo || key > pos) return -1;
    const int nth = P.page_shift >= 0 ? key >> P.page_shift : key / P.page_size;
    const int page = bt[nth];
    if (page < 0 || page >= P.num_pages) { qb_set_status(P.status, QB_STATUS_BAD_PAGE, page, 6); return -1; }
    return (page * P.nkv + kvh) * P.page_size + (key - nth * P.page_size);
  };
  // the copies of a round: half a warp a row of 256 bytes, the sixteen rows of K and then those of V
  __nv_bfloat16* mine = ring + (size_t)warp * DD_STAGES * DD_ROUND;
  const uint32_t mine_s = (uint32_t)__cvta_generic_to_shared(mine);
  const int piece = lane & 15, odd = lane >> 4;
  auto ask = [&](int at, int stage) {
    const uint32_t dst = mine_s + (uint32_t)stage * DD_ROUND * 2;
#pragma unroll
    for (int n = 0; n < DD_KEYS / 2; ++n) {
      const int i = 2 * n + odd, row = __shfl_sync(0xffffffffu, at, i);
      const size_t from = (size_t)max(row, 0) * DD_HD + piece * 8;
      dd_copy16(dst + (uint32_t)(i * 256 + ((piece ^ ((i & 1) << 2)) << 4)), k_cache + from, row >= 0);
      dd_copy16(dst + (uint32_t)(DD_KEYS * 256 + i * 256 + ((piece ^ (((i >> 1) & 3) << 1)) << 4)), v_cache + from, row >= 0);
    }
  };

  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  const int r0 = lo / DD_KEYS + rank * warps + warp;
  int at = place(r0);
  const int at1 = place(r0 + step);
  // the launch before writes the token's own key and value and its queries; the keys of the rounds before its own lie in the cache since
  // earlier steps and are asked for while that launch ends
  const bool e0 = P.early && r0 < last, e1 = P.early && r0 + step < last;      // the same for the whole warp
  if (e0) { ask(at, 0); commit(); }
  if (e1) { ask(at1, 1); commit(); }
  if (P.early) qb_follow();
  uint4 qa[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    qa[i] = g < G ? *reinterpret_cast<const uint4*>(q + ((size_t)tok * P.nq + kvh * G + g) * DD_HD + (t + 4 * i) * 8)
                  : make_uint4(0, 0, 0, 0);

  float m = -INFINITY, l = 0.f;                      // of head g: the maximum of all lanes, this lane's part of the sum
  float o[8][4];                                     // tile e: dims 8 g + e and 64 + 8 g + e of heads 2 t and 2 t + 1
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e][0] = o[e][1] = o[e][2] = o[e][3] = 0.f;
  auto use = [&](int stage, unsigned seen) {
    const __nv_bfloat16 *ks = mine + stage * DD_ROUND, *vs = ks + DD_KEYS * DD_HD;
    struct { uint4 k[2][4], v[4][2]; } x;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        x.k[n][i] = *reinterpret_cast<const uint4*>(ks + (g + 8 * n) * DD_HD + (((t + 4 * i) ^ ((g & 1) << 2)) << 3));
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int key = 2 * t + (n & 1) + 8 * (n >> 1);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        x.v[n][i] = *reinterpret_cast<const uint4*>(vs + key * DD_HD + (((g + 8 * i) ^ (((key >> 1) & 3) << 1)) << 3));
    }
    float s[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float s2[4] = {0.f, 0.f, 0.f, 0.f};            // two chains of four products
      s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dd_mma(s[n], qa[i].x, 0u, qa[i].y, 0u, x.k[n][i].x, x.k[n][i].y);
        dd_mma(s2, qa[i].z, 0u, qa[i].w, 0u, x.k[n][i].z, x.k[n][i].w);
      }
      s[n][0] += s2[0];
      s[n][1] += s2[1];
    }
    float top = -INFINITY;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float y = s[n][e] * scale_log2;
        if (SPLIT && P.cap > 0.f) y = P.cap * tanhf(s[n][e] * P.scale / P.cap) * LOG2E;
        s[n][e] = (seen >> (8 * n + 2 * t + e)) & 1u ? y : -INFINITY;
        top = fmaxf(top, s[n][e]);
      }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    const float m_new = fmaxf(m, top), ref = m_new == -INFINITY ? 0.f : m_new;
    const float corr = dd_exp2(m - ref);
    m = m_new;
    float sum = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[n][e] = dd_exp2(s[n][e] - ref);
        sum += s[n][e];
      }
    l = l * corr + sum;
    const float c0 = __shfl_sync(0xffffffffu, corr, 8 * t), c1 = __shfl_sync(0xffffffffu, corr, 8 * t + 4);
    const uint32_t b0 = dd_pack(s[0][0], s[0][1]), b1 = dd_pack(s[1][0], s[1][1]);
    uint32_t mid0 = 0u, mid1 = 0u, low0 = 0u, low1 = 0u;        // what the rounding left, and what is left of that: exact
    if (SPLIT) {
      auto left = [](float x, uint32_t part, int e) { return x - __uint_as_float(e ? part & 0xffff0000u : part << 16); };
      float r[4] = {left(s[0][0], b0, 0), left(s[0][1], b0, 1), left(s[1][0], b1, 0), left(s[1][1], b1, 1)};
      mid0 = dd_pack(r[0], r[1]);
      mid1 = dd_pack(r[2], r[3]);
      low0 = dd_pack(left(r[0], mid0, 0), left(r[1], mid0, 1));
      low1 = dd_pack(left(r[2], mid1, 0), left(r[3], mid1, 1));
    }
    if (__any_sync(0xffffffffu, corr != 1.f)) {      // a maximum has grown
#pragma unroll
      for (int e = 0; e < 8; ++e) { o[e][0] *= c0; o[e][1] *= c1; o[e][2] *= c0; o[e][3] *= c1; }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t sel = (e & 1) ? 0x7632u : 0x5410u;      // the upper or the lower bfloat16 of both keys' words
      auto word = [&](const uint4& w) { return (e >> 1) == 0 ? w.x : (e >> 1) == 1 ? w.y : (e >> 1) == 2 ? w.z : w.w; };
      const uint32_t a0 = __byte_perm(word(x.v[0][0]), word(x.v[1][0]), sel), a1 = __byte_perm(word(x.v[0][1]), word(x.v[1][1]), sel);
      const uint32_t a2 = __byte_perm(word(x.v[2][0]), word(x.v[3][0]), sel), a3 = __byte_perm(word(x.v[2][1]), word(x.v[3][1]), sel);
      dd_mma(o[e], a0, a1, a2, a3, b0, b1);
      if (SPLIT) {
        dd_mma(o[e], a0, a1, a2, a3, mid0, mid1);
        dd_mma(o[e], a0, a1, a2, a3, low0, low1);
      }
    }
  };

  auto which = [](int at) { return __ballot_sync(0xffffffffu, at >= 0) & 0xffffu; };
  unsigned now = which(at), next = which(at1);       // the keys of the round in use and of the one behind it
  if (!e0) { ask(at, 0); commit(); }
  if (!e1) { ask(at1, 1); commit(); }
  at = place(r0 + 2 * step);
  int stage = 0;
  for (int r = r0; r <= last; r += step) {           // the same for the whole warp
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();                                    // this round of every lane has landed, the one before has been read
    const unsigned after = which(at);
    ask(at, stage == 0 ? 2 : stage - 1);
    commit();
    at = place(r + 3 * step);
    use(stage, now);
    now = next;
    next = after;
    stage = stage == 2 ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                   // the rings become the place of the sums
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t == 0) { s_m[warp][g] = m; s_l[warp][g] = l; }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    s_o[warp][2 * t][8 * e + g] = o[e][0];
    s_o[warp][2 * t + 1][8 * e + g] = o[e][1];
    s_o[warp][2 * t][64 + 8 * e + g] = o[e][2];
    s_o[warp][2 * t + 1][64 + 8 * e + g] = o[e][3];
  }
  __syncthreads();
  // the warps of the block in order, then the blocks of the cluster in order; each block finishes its share of the numbers
  for (int i = tid; i < G * DD_HD; i += blockDim.x) {
    const int h = i / DD_HD, d = i % DD_HD;
    float top = -INFINITY;
    for (int w = 0; w < warps; ++w) top = fmaxf(top, s_m[w][h]);
    const float ref = top == -INFINITY ? 0.f : top;
    float sum = 0.f, x = 0.f;
    for (int w = 0; w < warps; ++w) {
      const float f = dd_exp2(s_m[w][h] - ref);
      sum = fmaf(s_l[w][h], f, sum);
      x = fmaf(s_o[w][h][d], f, x);
    }
    s_po[h][d] = x;
    if (d == 0) { s_pm[h] = top; s_pl[h] = sum; }
  }
  if (P.S > 1) dd_cluster_sync();
  else __syncthreads();
  for (int i = tid * P.S + rank; i < G * DD_HD; i += blockDim.x * P.S) {
    const int h = i / DD_HD, d = i % DD_HD;
    float x, sum;
    if (P.S > 1) {
      float top = -INFINITY;
      for (int c = 0; c < P.S; ++c) top = fmaxf(top, dd_remote(&s_pm[h], c));
      const float ref = top == -INFINITY ? 0.f : top;
      x = sum = 0.f;
      for (int c = 0; c < P.S; ++c) {
        const float f = dd_exp2(dd_remote(&s_pm[h], c) - ref);
        sum = fmaf(dd_remote(&s_pl[h], c), f, sum);
        x = fmaf(dd_remote(&s_po[h][d], c), f, x);
      }
    } else {
      x = s_po[h][d];
      sum = s_pl[h];
    }
    const int dim = (d & 64) + (d & 7) * 8 + ((d & 63) >> 3);
    out[((size_t)tok * P.nq + kvh * G + h) * DD_HD + dim] = __float2bfloat16_rn(sum == 0.f ? 0.f : x / sum);     // no key read: 0; a sum that is no number stays none
  }
  if (P.S > 1) dd_cluster_sync();                    // nobody leaves while its sums are read
}

}  // namespace

// 1 if the kernel takes these sizes.
extern "C" int qb_attn_decode_direct_supported(int nq, int nkv, int hd) {
  return hd == DD_HD && nkv > 0 && nq % nkv == 0 && nq / nkv <= 8 ? 1 : 0;
}

// Warps a block and blocks a unit (a (token, kv head)).  Eight warps a block and as many blocks a unit, up to eight, as fill the SMs once,
// but no more than the keys give rounds for; with more units than SMs blocks of four warps, two to an SM, a unit two of them where that
// leaves eight rounds a warp.
static void dd_shape(long units, int keys, int& warps, int& S) {
  const int rounds = (keys + DD_KEYS - 1) / DD_KEYS;
  warps = 8;
  S = 1;
  if (units >= 148) {
    warps = 4;
    S = units < 592 && rounds >= 64 ? 2 : 1;
  } else {
    // clusters fill a GPC of 16 to 20 SMs in part only: what does not fit waits for a second wave (48 units of 3 blocks: 32 us for 6 tokens
    // of 3,000 keys, 2 blocks 22)
    while (S < 6 && units * (S + 1) <= (S < 2 ? 148 : S < 4 ? 128 : 120)) ++S;
    if (units <= 12) S = 8;
  }
  while (S > 1 && (S - 1) * warps >= rounds) --S;
}
static int dd_keys(int longest, int window, int chunk) {
  const int keys = window > 0 && window < longest ? window : longest;
  return chunk > 0 && chunk < keys ? chunk : keys;
}

// Whether these single tokens, with `longest` and `total` keys, are faster here than in the kernel that takes all other shapes: the persistent
// one with its merge, whose blocks share the keys of all tokens alike, or for weights that stay 32-bit the one of attention_rows.cuh.  Here a
// unit's keys are walked by its own S blocks, so one long request among short ones, or few units, which eight blocks each do not make
// fill the SMs, cost what that walk costs: 8.0 us for 1,000 keys a block of eight warps.  The others' times are lines through what they
// measure; over 370 mixes of lengths the choice is 0.3 % off the better kernel on average, 17 % at most.  Measured on a B200, here / persistent, 48 + 8 heads: 16 tokens, one of 131,072 keys and the others of 500, 1,029 / 164 us, one of 8,000 69
// / 33, one of 2,000 23 / 25, all of 8,000 87 / 116; one of 131,072 140 / 119, of 24,000 33 / 37; 6 + 1 heads, one token of 131,072 141 / 62, of
// 24,000 31 / 52.
extern "C" int qb_attn_decode_direct_wins(int n_dec, int nq, int nkv, int hd, int longest, long long total, int window, int chunk,
                                          int two_part) {
  if (n_dec <= 0 || longest <= 0 || !qb_attn_decode_direct_supported(nq, nkv, hd)) return 0;
  const long units = (long)n_dec * nkv;
  const int keys = dd_keys(longest, window, chunk), G = nq / nkv;
  int warps, S;
  dd_shape(units, keys, warps, S);
  const double all = (double)(total < (long long)n_dec * keys ? (total > keys ? total : keys) : (long long)n_dec * keys) * nkv;
  const double here = (5.5 + 0.0080 * keys / S * 8 / warps) * (two_part ? 1.12 : 1.08);      // 1.08: the other kernel where they are close
  if (two_part) {
    const int groups = G % 4 == 0 ? G / 4 : G % 2 == 0 ? G / 2 : G;      // q heads of a kv head a block: 4, 2 or 1
    double ranges = 1184.0 / (units * (G / 4 > 1 ? G / 4 : 1));
    ranges = fmin(fmin(ranges, 64.0), (keys + 255) / 256);
    return here <= 12.0 + 2.8 / 64 * fmax(all * groups / 148, keys / fmax(ranges, 1.0)) ? 1 : 0;
  }
  const double segments = fmin(148.0 * keys / all, (keys + 63) / 64);     // that the longest pair is cut into: the merge adds them one by one
  return here <= 13.0 + all * (4 * DD_HD) / 5.0e6 + 0.2 * segments ? 1 : 0;
}

// dec_tok: the token rows of the n_dec single tokens; longest: keys of the longest request (an upper bound is enough).  early: the two
// launches before this one write no key or value but the tokens' own and neither the tables nor the tokens' places; the kernel then reads
// these before the launch before it has ended.
extern "C" int qb_attn_decode_direct(const void* q, const void* k_cache, const void* v_cache, void* out, const int* dec_tok, int n_dec,
                                     const int* tok_pos, const int* tok_req, const int* block_table, int bt_stride, int nq, int nkv,
                                     int hd, int page_size, int num_pages, float scale, int window, int longest, int two_part,
                                     float cap, int chunk, int early, int* status, cudaStream_t stream) {
  if (n_dec <= 0) return 0;
  if (chunk < 0 || (cap > 0.f && !two_part)) return QB_ERR_BAD_ARG;
  if (!qb_attn_decode_direct_supported(nq, nkv, hd) || page_size <= 0) return QB_ERR_UNSUPPORTED;
  if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) != 0) return QB_ERR_UNSUPPORTED;
  int shift = -1;
  for (int i = 0; i < 31; ++i)
    if (page_size == 1 << i) shift = i;
  const long units = (long)n_dec * nkv;
  if (units * 8 > 0x7fffffffL || (long)num_pages * nkv * page_size > 0x7fffffffL) return QB_ERR_UNSUPPORTED;
  // This kernel and the persistent one with its merge launch, contexts of like length, 48 + 8 heads: one token of 60 keys 5.5 and 10.8 us, of
  // 2,100 10.0 and 15.8; 2 of 24,000 and 18,000 42 and 48 (four blocks a unit 53), 4 of 4,000 19 and 29, 8 of 2,100 to 1,050 18 and 26,
  // 16 of 2,000 27 and 40, 64 of 500 33 and 49, of 2,100 to 1,050 91 to 95 and 100.  `two_part`: weights in parts (SPLIT).
  int warps, S;
  dd_shape(units, dd_keys(longest, window, chunk), warps, S);
  const DecodeArgs P{dec_tok, tok_pos, tok_req, block_table, bt_stride, nq, nkv, page_size, shift, num_pages, window, chunk, S,
                     early, scale, cap, status};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units * S));
  cfg.blockDim = dim3((unsigned)(warps * 32));
  cfg.dynamicSmemBytes = (size_t)warps * DD_STAGES * DD_ROUND * sizeof(__nv_bfloat16);      // more than the sums want
  cfg.stream = stream;
  auto kern = two_part ? attn_decode_direct_kernel<true> : attn_decode_direct_kernel<false>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DD_MAX_WARPS * DD_STAGES * DD_ROUND * 2);
  if (err != cudaSuccess) return (int)err;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see qb_follow
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)S;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = S > 1 ? 2 : 1;
  err = cudaLaunchKernelEx(&cfg, kern, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_cache,
                                             (const __nv_bfloat16*)v_cache, (__nv_bfloat16*)out, P);
  if (err != cudaSuccess) return (int)err;
  QB_LAUNCH_CHECK();
  return 0;
}
