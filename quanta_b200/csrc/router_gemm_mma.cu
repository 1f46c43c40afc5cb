// Router logits of many tokens on the tensor cores, to float32 accuracy:
//   logits[t, e] = sum_k x[t, k] * gate[e, k],  x bfloat16, gate float32.
//
// The float32 gate is held as THREE bfloat16 matrices hi + mid + lo (each the bfloat16 rounding of what
// the ones before leave over: 3 x 8 mantissa bits carry the 24 of a float32), so every product
// x * piece is exact in float32 and the sum runs in float32 accumulators.  The inner
// dimension is taken in chunks of 64: a chunk's sum starts from zero and is then added to the running
// total, in chunk order, whatever the number of tokens, so a token's logits do not depend on the step.
// The inner dimension is also cut into ranges of RG_KSPLIT (a constant), one block a range, whose sums
// come out side by side, [ranges][T][E]; the selection kernel adds them in range order.
// (src/quanta/minimax/moe.py:44, "logits = fp32(x) @ fp32(gate).T".)  Prompt portions use this kernel;
// steps of few tokens keep the SIMT kernel, which reads the float32 gate once.
//
// A work item is 128 experts x NT tokens of one range: tcgen05.mma with the experts as M and the tokens as N.  One warp copies by TMA, a
// stage the three pieces' tiles and the tokens'; one issues twelve MMAs a chunk into one of two accumulators; eight add the finished
// chunk, read from TMEM, to the totals in their registers while the next runs, and write these at an item's end, under the next item's
// MMAs.  Bound by how many bytes of the next chunks can be on their way beside the one in work (three stages of up to 72 KB: the tensor
// cores are busy 55 % of a block's time, L2 22 %).  256 experts of 3,072: 300 tokens 28.7 -> 14.4 us, 2,048 45 -> 18.4, 12,800 (60 GFLOP)
// 210 -> 64; 768 of 6,144, 4,000 tokens 395 -> 103 (mma.sync from shared memory before; a block an item without the overlap: 81 us for the
// 12,800).
// Needs K % 8 == 0 (16-byte rows).
#include <climits>

#include "tensor_core.cuh"

namespace {

constexpr int RG_M = 128;           // experts a block
constexpr int RG_KSPLIT = 768;      // inner-dimension range of one block: a multiple of TC_BK
constexpr int RG_ADD_WARPS = 8, RG_THREADS = 32 * (RG_ADD_WARPS + 2);
constexpr uint32_t RG_W_BYTES = RG_M * TC_BK * 2;      // a piece's tile
__host__ __device__ constexpr uint32_t rg_stage_bytes(int nt) { return 3 * RG_W_BYTES + (uint32_t)nt * TC_BK * 2; }
constexpr int RG_STAGES = 3;       // 168, 192 or 216 KB

struct RgShared {
  uint64_t full[RG_STAGES], empty[RG_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

// tm_x: x [T, K], boxes [NT][64]; tm_w: the pieces [3][E][K], boxes [1][128][64]
template <int NT>
__global__ void __launch_bounds__(RG_THREADS, 1)
router_gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, float* __restrict__ logits,
                      int T, int E, int K, int tiles, int blocks_e, int items, int* status) {
  constexpr int STAGES = RG_STAGES, COLS = NT / 2;      // a warp adds half of the tokens, of 32 experts
  constexpr uint32_t STAGE = rg_stage_bytes(NT), TMEM_COLS = NT == 192 ? 512 : 2 * NT;      // (a power of two)
  extern __shared__ unsigned char rg_smem[];
  __shared__ RgShared sh;
  const uint32_t ring = (smem_u32(rg_smem) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &sh.abort_flag;
  // work item -> its first token, expert and k, and its chunks; the items that run at the same time share a range of the pieces
  auto place = [&](int item, int& t0, int& e0, int& k0) {
    t0 = item % tiles * NT;
    e0 = item / tiles % blocks_e * RG_M;
    k0 = item / tiles / blocks_e * RG_KSPLIT;
    return (min(K - k0, RG_KSPLIT) + TC_BK - 1) / TC_BK;
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh.full[s]), 1);
      mbar_init(smem_u32(&sh.empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh.acc_full[b]), 1);
      mbar_init(smem_u32(&sh.acc_empty[b]), RG_ADD_WARPS);
    }
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == RG_ADD_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&sh.tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem_base;

  if (warp == RG_ADD_WARPS + 1) {
    // ---------------- copies ----------------
    if (lane == 0) {
      const uint64_t keep = l2_policy_evict_last();
      int armed = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int t0, e0, k0;
        const int chunks = place(item, t0, e0, k0);
        for (int i = 0; i < chunks; ++i) {
          const int c = armed, s = c % STAGES;
          const uint32_t st = ring + (uint32_t)s * STAGE, full = smem_u32(&sh.full[s]);
          ok = c < STAGES || mbar_wait(smem_u32(&sh.empty[s]), (uint32_t)(c / STAGES - 1) & 1u, abort_flag);
          if (!ok) break;
          mbar_expect_tx(full, STAGE);
          tma_load_2d(st + 3 * RG_W_BYTES, &tm_x, k0 + i * TC_BK, t0, full, keep);
          for (int p = 0; p < 3; ++p) tma_load_3d(st + p * RG_W_BYTES, &tm_w, k0 + i * TC_BK, e0, p, full, keep);
          armed = c + 1;
        }
      }
      if (*abort_flag) {      // let the copies that were issued land before the shared memory is given away
        for (int c = max(0, armed - STAGES); c < armed; ++c) {
          const uint64_t ns = global_ns();
          for (uint32_t it = 0; it < TC_SPIN_LIMIT && !mbar_try_wait(smem_u32(&sh.full[c % STAGES]), (uint32_t)(c / STAGES) & 1u); ++it)
            if ((it & 63u) == 63u && global_ns() - ns > TC_WAIT_NS) break;
        }
      }
    }
  } else if (warp == RG_ADD_WARPS) {
    // ---------------- MMAs ----------------
    if (lane == 0) {
      int c = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int t0, e0, k0;
        const int chunks = place(item, t0, e0, k0);
        const uint32_t idesc = umma_idesc(RG_M, min(NT, (T - t0 + 15) & ~15));
        for (int i = 0; i < chunks; ++i, ++c) {
          const int s = c % STAGES, b = c & 1;
          ok = (c < 2 || mbar_wait(smem_u32(&sh.acc_empty[b]), (uint32_t)(c / 2 - 1) & 1u, abort_flag)) &&
               mbar_wait(smem_u32(&sh.full[s]), (uint32_t)(c / STAGES) & 1u, abort_flag);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = ring + (uint32_t)s * STAGE;
          const uint64_t xd = umma_desc_sw128(st + 3 * RG_W_BYTES);
#pragma unroll
          for (int k16 = 0; k16 < TC_BK / 16; ++k16)
#pragma unroll
            for (int p = 0; p < 3; ++p)      // hi, then mid, then lo; 16 k elements: 32 bytes along the swizzled row
              umma_bf16(tmem + (uint32_t)(b * NT), umma_desc_sw128(st + p * RG_W_BYTES) + (uint64_t)(2 * k16), xd + (uint64_t)(2 * k16),
                        idesc, k16 + p != 0 ? 1u : 0u);
          umma_commit(smem_u32(&sh.empty[s]));
          umma_commit(smem_u32(&sh.acc_full[b]));
        }
      }
    }
  } else {
    // ---------------- totals: the chunks' sums in chunk order.  A warp reaches the 32 TMEM lanes of its index modulo 4 ----------------
    const int quarter = warp & 3, col0 = (warp >> 2) * COLS;
    const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
    int c = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      int t0, e0, k0;
      const int chunks = place(item, t0, e0, k0);
      float total[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) total[i] = 0.f;
      for (int i = 0; i < chunks && ok; ++i, ++c) {
        const int b = c & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh.acc_full[b]), (uint32_t)(c / 2) & 1u, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int j = 0; j < COLS; j += 32) {
          uint32_t v0[16], v1[16];
          tmem_ld16(at + (uint32_t)(b * NT + j), v0);
          tmem_ld16(at + (uint32_t)(b * NT + j + 16), v1);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            total[j + u] += __uint_as_float(v0[u]);
            total[j + 16 + u] += __uint_as_float(v1[u]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sh.acc_empty[b])) : "memory");
      }
      if (!ok) {      // a wait ran out: the sums that are missing are no numbers, for callers without status words too
#pragma unroll
        for (int i = 0; i < COLS; ++i) total[i] = __int_as_float(0x7fffffff);
      }
      const int e = e0 + quarter * 32 + lane, n = T - t0 - col0;      // this warp's tokens (none or fewer than COLS: nothing there)
      if (e < E) {
        float* dst = logits + ((size_t)(k0 / RG_KSPLIT) * T + t0 + col0) * E + e;
#pragma unroll
        for (int i = 0; i < COLS; ++i)
          if (i < n) dst[(size_t)i * E] = total[i];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == RG_ADD_WARPS)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  if (threadIdx.x == 0 && sh.abort_flag && status != nullptr) qb_set_status(status, QB_STATUS_WAIT_TIMEOUT, (int)blockIdx.x, 10);
}

// out[p][i] = the p-th bfloat16 piece of w[i]: hi, mid, lo
__global__ void split3_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float v = w[i];
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(mid);
    out[i] = hi;
    out[n + i] = mid;
    out[2 * n + i] = __float2bfloat16_rn(r2);
  }
}

}  // namespace

// w float32 [n] -> out bfloat16 [3][n]
extern "C" int qb_split3_bf16(const float* w, void* out, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  split3_kernel<<<blocks, 256, 0, stream>>>(w, (__nv_bfloat16*)out, (size_t)n);
  QB_LAUNCH_CHECK();
  return 0;
}

// how many ranges the inner dimension is cut into: the first size of the logits
extern "C" int qb_router_gemm_mma_parts(int K) { return K <= 0 ? 0 : (K + RG_KSPLIT - 1) / RG_KSPLIT; }

// x bf16 [T, K]; pieces bf16 [3, E, K] (qb_split3_bf16 of the float32 gate); logits float32 [parts, T, E]; status may be null
extern "C" int qb_router_gemm_mma(const void* x, const void* pieces, float* logits, int T, int E, int K, int* status,
                                  cudaStream_t stream) {
  if (T <= 0 || E <= 0) return 0;
  if (K <= 0 || K % 8) return QB_ERR_UNSUPPORTED;
  if ((((uintptr_t)x | (uintptr_t)pieces) & 15) != 0) return QB_ERR_UNSUPPORTED;
  int sms = 0;
  int rc = sm_count(sms);
  if (rc) return rc;
  const int blocks_e = (E + RG_M - 1) / RG_M, parts = (K + RG_KSPLIT - 1) / RG_KSPLIT;
  // The token tile by the rounds of items over the SMs times an item's time, which goes with the bytes of its stages and its products, 1 + NT / 64
  // (7, 10.5 and 14 us of 768 k).  256 experts of 3,072, tiles of 64 / 128 / 192: 300 tokens 14.4 / 18.4 / - us, 2,048 22.5 / 18.5 / 22.5, 4,096
  // 38.9 / 29.7 / 36.9, 12,800 94 / 70 / 64, 16,384 117 / 81 / 78 (256 in a ring of two stages: 28.7, 71 and 87 for the last three).
  const auto blocks = [&](int nt) { return (long long)blocks_e * parts * ((T + nt - 1) / nt); };
  const auto cost = [&](int nt) { return ((blocks(nt) + sms - 1) / sms) * (1 + nt / 64); };
  const int nt = cost(64) <= cost(128) && cost(64) <= cost(192) ? 64 : cost(128) <= cost(192) ? 128 : 192;
  CUtensorMap tm_x, tm_w;
  rc = map_2d(&tm_x, x, (uint64_t)T, (uint64_t)K, (uint32_t)nt);
  if (rc) return rc;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)E, 3}, strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)E * K * 2};
  const cuuint32_t box[3] = {TC_BK, RG_M, 1};
  rc = make_map(&tm_w, pieces, 3, dims, strides, box);
  if (rc) return rc;
  if (blocks(nt) > INT_MAX) return QB_ERR_UNSUPPORTED;
  const int items = (int)blocks(nt), grid = items < sms ? items : sms;
  const size_t smem = (size_t)RG_STAGES * rg_stage_bytes(nt) + 1024;
#define QB_RG(NT_)                                                                                                              \
  do {                                                                                                                          \
    cudaError_t err = cudaFuncSetAttribute(router_gemm_tc_kernel<NT_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
    if (err != cudaSuccess) return (int)err;                                                                                    \
    router_gemm_tc_kernel<NT_><<<grid, RG_THREADS, smem, stream>>>(tm_x, tm_w, logits, T, E, K, (T + nt - 1) / nt, blocks_e, items, status);                       \
  } while (0)
  if (nt == 64) QB_RG(64);
  else if (nt == 128) QB_RG(128);
  else QB_RG(192);
#undef QB_RG
  QB_LAUNCH_CHECK();
  return 0;
}
