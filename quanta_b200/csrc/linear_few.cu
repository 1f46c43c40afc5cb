// out[r] = x[r] W^T for a few bfloat16 rows: the projections, dense feed-forwards and output matrices of a step that decodes.
//
// Bound by the bytes of W.  A block takes 16 rows of W, its eight warps 64 numbers of the inner dimension in turn.  A lane loads the 16
// numbers of a row's 128 bytes that it then multiplies (the order of the inner dimension inside an mma is free as long as both operands
// have it), 32 bytes a load, so that weights go from memory to registers without shared memory or a barrier: up to 128 KB on
// their way an SM, of which 45 keep the memory busy.  Between the launches of a step the library's kernels wait for the launch before
// them and then for their first weights; here, where the caller allows it (`early`), blocks are placed while the launch before runs and ask
// for their first pieces before they wait for it, and the products follow the arrival of x.  That pays behind launches that are one
// short chain of reads (8 requests, a delta rule's model: 637 us for two steps without, 603 with it), not behind those that
// use the memory or fill the SMs themselves (an attention, the norm over eight experts' slots: the blocks slow them and fall unevenly
// on the SMs that are left; 8 requests of the M2-family sizes 2,518 us with, 2,474 without).  x is read by every block: out of L1 after the SM's
// first where its rows fit there (8 rows of 8,192 do), else out of L2.  A row's sums are taken in an order that depends on K alone.
//
// Measured on a B200, one product after another in a graph, weights from memory, microseconds (library: at 32 rows, its fastest kernel):
//   [N, K]            bytes at 6.5 TB/s   library   8 rows   16 rows   32 rows
//   8,192 x 3,072            7.7            11.4      9.1      10.8      14.6
//   3,072 x 6,144            5.8            11.2      7.7       8.8      13.0
//   32,000 x 2,048          20.0            27.0     21.3      24.7      36.1
//   2,048 x 5,632            3.5             9.9      6.2       7.5       8.2
//   2,048 x 2,048            1.3             5.5      2.2       2.8       3.6
//   3,072 x 768              0.7             4.2      1.8       2.0       2.6
// Whole decode steps (graph, 1,000 keys; library for all / for the larger matrices only / this for all up to 32 rows): four layers of the
// M2-family sizes, 1 request 398 / 398 / 381 us, 24 2,679 / 2,678 / 2,720, 32 3,144 / 3,112 / 3,142; six layers of width 2,048 with delta rules, 1
// request 313 / 269 / 233, 16 352 / 315 / 304, 20 362 / 335 / 350, 32 395 / 376 / 398; with three recurrences, 16 589 / 551 / 542, 20 718 / 685 / 721.
#include "common.cuh"

constexpr int LF_WARPS = 8;
constexpr int LF_KB = 64;                // numbers of the inner dimension a warp takes at a time: 128 bytes of each row of W

struct LinearFew {
  const __nv_bfloat16 *x, *w;
  void* out;
  int rows, K, N;
};

struct alignas(32) LfPiece {
  uint32_t u[8];
};

__device__ __forceinline__ LfPiece lf_stream(const __nv_bfloat16* p) {       // read once: not kept in L1
  LfPiece v;
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.u[0]), "=r"(v.u[1]), "=r"(v.u[2]), "=r"(v.u[3]), "=r"(v.u[4]), "=r"(v.u[5]), "=r"(v.u[6]), "=r"(v.u[7])
               : "l"(p));
  return v;
}

__device__ __forceinline__ LfPiece lf_load(const __nv_bfloat16* p) {
  LfPiece v;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.u[0]), "=r"(v.u[1]), "=r"(v.u[2]), "=r"(v.u[3]), "=r"(v.u[4]), "=r"(v.u[5]), "=r"(v.u[6]), "=r"(v.u[7])
               : "l"(p));
  return v;
}

__device__ __forceinline__ void lf_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: tiles of 8 input rows.  D, XD: pieces of W and of x a warp holds ahead.  GLU: W is [gate; up] of N features each, a block takes 8 rows of
// both, and out = silu(gate) * up of the sums, each rounded to bfloat16 first (what a product and an activation kernel leave).
template <int NT, int D, int XD, int MINB, bool GLU, typename O>
__global__ void __launch_bounds__(LF_WARPS * 32, MINB) linear_few_kernel(LinearFew a, int early) {
  static_assert(D % XD == 0, "the ring of x divides the ring of W");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  constexpr int FEATS = GLU ? 8 : 16;
  const int n0 = blockIdx.x * FEATS;
  const int kbs = (a.K + LF_KB - 1) / LF_KB;
  const __nv_bfloat16* wr[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) wr[h] = a.w + (size_t)(GLU ? min(n0 + g, a.N - 1) + h * a.N : min(n0 + h * 8 + g, a.N - 1)) * a.K + t * 16;
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xr[n] = a.x + (size_t)min(n * 8 + g, a.rows - 1) * a.K + t * 16;
  const LfPiece none = {};
  LfPiece wb[D][2], xb[XD][NT];
  auto fetch_w = [&](int kb, LfPiece (&b)[2]) {
    const bool in = kb < kbs && kb * LF_KB + t * 16 < a.K;
#pragma unroll
    for (int h = 0; h < 2; ++h) b[h] = in ? lf_stream(wr[h] + kb * LF_KB) : none;
  };
  auto fetch_x = [&](int kb, LfPiece (&b)[NT]) {
    const bool in = kb < kbs && kb * LF_KB + t * 16 < a.K;
#pragma unroll
    for (int n = 0; n < NT; ++n) b[n] = in ? lf_load(xr[n] + kb * LF_KB) : none;
  };
#pragma unroll
  for (int d = 0; d < D; ++d) fetch_w(warp + d * LF_WARPS, wb[d]);
  if (early) qb_follow();         // (a launch that is not early starts behind the one before it)
#pragma unroll
  for (int d = 0; d < XD; ++d) fetch_x(warp + d * LF_WARPS, xb[d]);
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
  for (int k0 = warp; k0 < kbs; k0 += D * LF_WARPS) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int kb = k0 + d * LF_WARPS;
      if (kb >= kbs) break;
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int n = 0; n < NT; ++n)
          lf_mma(acc[n], wb[d][0].u[2 * s], wb[d][1].u[2 * s], wb[d][0].u[2 * s + 1], wb[d][1].u[2 * s + 1],
                 xb[d % XD][n].u[2 * s], xb[d % XD][n].u[2 * s + 1]);
      fetch_w(kb + D * LF_WARPS, wb[d]);
      fetch_x(kb + XD * LF_WARPS, xb[d % XD]);
    }
  }
  // the warps' parts, added in the order of the warps
  constexpr int ROWS = 16, PAD = ROWS + 4, TOK = NT * 8;
  __shared__ float part[LF_WARPS][TOK][PAD];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[warp][n * 8 + 2 * t + (i & 1)][g + 8 * (i >> 1)] = acc[n][i];
  __syncthreads();
  auto sum = [&](int tok, int row) {
    float s = part[0][tok][row];
#pragma unroll
    for (int w = 1; w < LF_WARPS; ++w) s += part[w][tok][row];
    return s;
  };
  for (int v = threadIdx.x; v < TOK * FEATS; v += LF_WARPS * 32) {
    const int tok = v / FEATS, row = v % FEATS;
    if (tok >= a.rows || n0 + row >= a.N) continue;
    float s = sum(tok, row);
    if (GLU) {
      const float gate = __bfloat162float(__float2bfloat16_rn(s)), up = __bfloat162float(__float2bfloat16_rn(sum(tok, row + 8)));
      s = gate / (1.f + expf(-gate)) * up;
    }
    reinterpret_cast<O*>(a.out)[(size_t)tok * a.N + n0 + row] = qb_from_float<O>(s);
  }
}

template <int NT, int D, int XD, int MINB>
static int linear_few_launch(const LinearFew& a, int out_dtype, bool glu, int early, cudaStream_t stream) {
  if (glu) {
    const int grid = (a.N + 7) / 8;
    if (early) qb_launch(linear_few_kernel<NT, D, XD, MINB, true, __nv_bfloat16>, grid, LF_WARPS * 32, 0, stream, a, 1);
    else linear_few_kernel<NT, D, XD, MINB, true, __nv_bfloat16><<<grid, LF_WARPS * 32, 0, stream>>>(a, 0);
    QB_LAUNCH_CHECK();
    return 0;
  }
  const int grid = (a.N + 15) / 16;
  if (early) QB_DISPATCH_DTYPE(out_dtype, O, qb_launch(linear_few_kernel<NT, D, XD, MINB, false, O>, grid, LF_WARPS * 32, 0, stream, a, 1));
  else QB_DISPATCH_DTYPE(out_dtype, O, (linear_few_kernel<NT, D, XD, MINB, false, O><<<grid, LF_WARPS * 32, 0, stream>>>(a, 0)));
  QB_LAUNCH_CHECK();
  return 0;
}

// Whether products of up to 32 rows of [N, K] are this kernel's: by the matrix alone, so that a row's numbers are the same in every step of up
// to 32 rows (the library's products run at 32 rows up to there).  It is the faster one up to 16 rows, and up to 32 where the matrix has a
// block an SM at most; in larger ones the mma.sync products of 17 to 32 rows and their reads of x take longer than the weights' bytes, which
// longer rows make worse.  Library / this, plain launches, microseconds: 3,072 x 8,192 14.5 / 11.3 at 8 rows, 14.6 / 18.8 at 32 (taken); 3,072 x
// 12,288 19.9 / 15.2 and 19.8 / 27.3, 8,192 x 12,288 36.4 / 33.0 and 36.6 / 53.5 (not); one block an SM: 1,024 x 12,288 20.8 / 10.0 and 20.8 / 16.1
// (taken), 2,048 x 16,384 20.7 / 16.2 and 21.0 / 23.3 (not).
extern "C" int qb_linear_few_takes(int rows, int K, int N) {
  return rows > 0 && rows <= 32 && K >= LF_KB && K % 16 == 0 && N > 0 && K <= ((N + 15) / 16 <= 148 ? 12288 : 8192);
}

// K a multiple of 16; x and w on 32 bytes.  early: W was written two launches before this one at the latest (or by the host), so that
// its first pieces are read before the launch before this one has ended.
static int linear_few_any(const LinearFew& a, int out_dtype, bool glu, int early, cudaStream_t stream) {
  const int rows = a.rows, N = glu ? 2 * a.N : a.N;
  if (rows <= 0 || N <= 0) return 0;
  if (a.K <= 0 || a.K % 16 || ((uintptr_t)a.x & 31) || ((uintptr_t)a.w & 31)) return QB_ERR_BAD_ARG;
  if (rows > 32) return QB_ERR_UNSUPPORTED;
  if (rows <= 8) return linear_few_launch<1, 4, 4, 2>(a, out_dtype, glu, early, stream);
  if (rows <= 16) return linear_few_launch<2, 4, 2, 2>(a, out_dtype, glu, early, stream);
  if ((N + 15) / 16 <= 148) return linear_few_launch<4, 4, 2, 1>(a, out_dtype, glu, early, stream);
  return linear_few_launch<4, 2, 1, 2>(a, out_dtype, glu, early, stream);
}

extern "C" int qb_linear_few(const void* x, const void* w, void* out, int out_dtype, int rows, int K, int N, int early,
                             cudaStream_t stream) {
  return linear_few_any(LinearFew{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, rows, K, N}, out_dtype, false, early, stream);
}

// out [rows, I] bfloat16 = silu(x W[:I]^T) * (x W[I:]^T), W [2 I, K]
extern "C" int qb_linear_few_silu(const void* x, const void* w, void* out, int rows, int K, int I, int early, cudaStream_t stream) {
  return linear_few_any(LinearFew{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, rows, K, I}, QB_BF16, true, early, stream);
}
