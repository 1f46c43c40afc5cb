// Routed experts on the 5th-generation tensor cores: TMA-fed tcgen05.mma with accumulators in TMEM.
//
// One block = one tile of up to NT token rows of ONE expert x 128 of its output features.  The
// expert's WEIGHTS are the 128-row operand (M = 128) and the token rows are the N operand ("swap
// A/B"), so an expert with few rows still uses the full height of the MMA and its weights stream
// through shared memory exactly once per token tile:
//
//   warp 0   : TMA producer.  Per 64-wide k block: weight tile(s) [128 x 64] and token tile [NT x 64],
//              bfloat16, 128-byte swizzle, into a ring of shared-memory stages (mbarrier expect_tx); lane 0
//              fetches the boxes, all lanes share the rows where the token rows are fetched one by one.
//   warp 1   : MMA issuer.  4 x tcgen05.mma (K = 16 each) per stage and matrix, D[128 x NT] float32 in
//              TMEM; tcgen05.commit frees the stage and, at the end, signals the epilogue.
//   warps 2-5: epilogue (2-9 in the blocks of a pair).  tcgen05.ld (one TMEM lane = one output feature per thread), then
//              MODE 1: act[p, j] = silu(gate) * up  (bfloat16),  gate/up = two accumulators; or, with the
//              clamped activation (EgAct), the routing weight applied to both accumulators first;
//              MODE 2: y[pair(p), n] = w[pair(p)] * acc  (float32);
//              MODE 3: act[p, j] = relu(acc)^2  (bfloat16): the first product of ungated experts, whose weights
//              are one matrix [E, I, K] (token rows fetched as in MODE 1, weight tiles laid out as in MODE 2).
//   (src/quanta/minimax/moe.py:59-88; rows p sorted by expert, see the plan kernels.)
//
// The token rows are read in p order: MODE 1 reads a gathered copy of x (gather kernel below) as one box a
// stage, or, for steps of few rows an expert, the rows of x themselves (gather_k), a box of one row each or
// four rows an instruction (EG_FOUR_ROWS);
// MODE 2 reads the act rows MODE 1 wrote.  Rows past the expert's last row compute garbage
// that the epilogue drops; TMA zero-fills past the end of a tensor, so K need not be a multiple of 64
// (it must be a multiple of 8: 16-byte rows).  No multicast: every tile comes from this GPU's memory through
// a plain per-block TMA load.  Tiles of 256 token rows are taken by two blocks together (see PAIR below).
//
// Every wait on an mbarrier is bounded; when one runs out the block records it in the status words,
// lets its copies in flight land, frees its TMEM and returns.
#include "tensor_core.cuh"

namespace {

constexpr int EG_M = 128;            // output features per block (UMMA M)
// Token tiles of more rows than this fetch their rows four an instruction (a box of one row costs the producer warp as much issue as
// four gathered ones, and from some 64 rows a stage on that is what the tensor cores wait for); smaller tiles, which wait for the weights,
// took the same time either way and keep the rows past the expert's last out of the copy.
constexpr int EG_FOUR_ROWS = 32;
constexpr int EG_BK = TC_BK;         // k elements per stage
constexpr int EG_THREADS = 192;        // producer warp, MMA warp, four epilogue warps
constexpr int EG_PAIR_THREADS = 320;   // a pair's blocks: eight epilogue warps

// silu(g) * u.  The exponential and the quotient are the fast ones (2 ulp); the result is rounded to bfloat16.
__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

// The activation of a gated first product (MODE 1).  kind 0: silu(gate) * up.  kind 1: the row's routing weight w
// multiplies both accumulators first (the expert reads w * x, and the products are linear in x), then
// g = min(w gate, limit), u = clamp(w up, -limit, limit), g * sigmoid(alpha g) * (u + 1).
struct EgAct {
  int kind;
  float limit, alpha;
};
__device__ __forceinline__ float clamped_glu(float g, float u, float w, const EgAct& a) {
  g = fminf(g * w, a.limit);
  u = fminf(fmaxf(u * w, -a.limit), a.limit);
  return __fdividef(g, 1.f + __expf(-a.alpha * g)) * (u + 1.f);
}

struct EgShared {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tmem_full;
  uint32_t tmem_base;
  int abort_flag;
};

// NM: weight tiles of 128 features a block (accumulators side by side in TMEM).  MODE 1 has two by its nature
// (gate and up rows of the same features).  MODE 2 takes two neighbouring blocks of 128 features when the
// token tile is 256 rows (steps bound by the tensor cores): the token tile, half of what a stage holds then,
// is fetched from L2 once for 256 features instead of once for 128.
//
// PAIR: two blocks on neighbouring SMs (a cluster of two) take one tile of 256 token rows together, each
// 128 (MODE 1) or 256 (MODE 2) of its features: tcgen05.mma.cta_group::2 with M = 256.  Each block fetches
// its own weight tiles and HALF of the token tile, and the tensor cores of both read both halves, so a block
// takes three quarters of the bytes from L2, and reads two thirds of the bytes from its shared memory, that
// it would alone.  The first block of the pair issues all MMAs; every copy of either block counts on the
// first block's barrier; a commit frees the stage in both.
//
// KS: slabs of 64 k a stage.  Two (launches of so few blocks that each streams its weights at the pace of its producer) come by one copy
// a matrix: the maps have the slab as a dimension of its own, and with HALF also gate / up and the expert, so that the copy
// leaves [slab][128 rows][64].
template <int MODE, int NM, bool PAIR, int KS>
__device__ __forceinline__ void
expert_gemm_tc_body(const CUtensorMap& tm_w, const CUtensorMap& tm_x,
                    void* __restrict__ out, const int* sorted_pair, const float* pair_w, const int* plan,
                    const int* tile_expert, const int* tile_row0, int E, int K, int N_out, int NT, int stages,
                    int tmem_cols, int gather_k, int* status, EgAct act, int early) {
  if (!early) qb_follow();
  constexpr bool HALF = MODE == 1 && NM == 1;              // 64 gate and 64 up rows in one weight tile
  constexpr int FEATS = HALF ? EG_M / 2 : MODE == 1 ? EG_M : NM * EG_M;      // output features a block
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;     // 0: the block that issues the MMAs
  extern __shared__ unsigned char smem_dyn[];
  // stage buffers need 1024-byte alignment for the 128-byte swizzle
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  __shared__ EgShared sh;
  __shared__ int s_pair[256];
  __shared__ float s_w[256];

  // (from L2: an early block has not waited yet)
  const int num_tiles = __ldcg(plan + 3 * E + 1);
  const int tile = blockIdx.y;
  if (tile >= num_tiles) {
    if (early) qb_follow();
    return;
  }
  const int e = __ldcg(tile_expert + tile), row0 = __ldcg(tile_row0 + tile);
  const int rows = min(NT, __ldcg(plan + 2 * E + e + 1) - row0);          // valid token rows of this tile
  const int j0 = blockIdx.x * FEATS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the MMA's N is what this tile holds, in steps of 16: an expert's last tile of a few rows costs the
  // tensor cores a few columns, not a whole tile (the box that TMA fetches keeps its size)
  const int n_mma = min(NT, (rows + 15) & ~15);
  // a pair's block holds half of the MMA's token rows: rows [rank * n_mma / 2, +n_mma / 2) of the tile, as
  // the first rows of a box of NT / 2
  constexpr int BK = KS * EG_BK;
  constexpr uint32_t A_SLAB = EG_M * EG_BK * 2, a_bytes = KS * A_SLAB;
  const uint32_t b_slab = (uint32_t)(PAIR ? NT / 2 : NT) * EG_BK * 2, b_bytes = KS * b_slab;
  const uint32_t stage_bytes = NM * a_bytes + b_bytes;
  const int k_blocks = (K + BK - 1) / BK;
  volatile int* abort_flag = &sh.abort_flag;
  const int w_row = MODE == 1 ? e * 2 * N_out + j0 : e * N_out + j0;
  const int ahead = MODE == 2 && !PAIR && early ? min(stages, k_blocks) : 0;      // k blocks whose weights are fetched before the wait

  // the second weight tile: the up rows of the same features, or the next 128 features (rows past the
  // expert's last are another expert's and give columns that the epilogue drops)
  const int w_row2 = w_row + (MODE == 1 ? N_out : EG_M);
  auto load_weights = [&](int kb, uint32_t st, uint32_t bar, uint64_t pol) {
    if constexpr (PAIR) {
      tma_load_2d_pair(st, &tm_w, kb * EG_BK, w_row, bar, pol);
      if (NM == 2) tma_load_2d_pair(st + a_bytes, &tm_w, kb * EG_BK, w_row2, bar, pol);
    } else if constexpr (KS == 2 && HALF) {
      tma_load_5d(st, &tm_w, 0, j0, 0, kb * KS, e, bar, pol);
    } else if constexpr (KS == 2) {
      tma_load_3d(st, &tm_w, 0, w_row, kb * KS, bar, pol);
    } else {
      tma_load_2d(st, &tm_w, kb * EG_BK, w_row, bar, pol);
      if (HALF) tma_load_2d(st + a_bytes / 2, &tm_w, kb * EG_BK, w_row2, bar, pol);
      if (NM == 2) tma_load_2d(st + a_bytes, &tm_w, kb * EG_BK, w_row2, bar, pol);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&sh.full[s]), 1);
      mbar_init(smem_u32(&sh.empty[s]), 1);
    }
    mbar_init(smem_u32(&sh.tmem_full), 1);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // an early block's first weights are on their way while the launch before it ends
    for (int kb = 0; kb < ahead; ++kb) {
      const uint32_t full = smem_u32(&sh.full[kb]);
      mbar_expect_tx(full, NM * a_bytes + b_bytes);
      load_weights(kb, smem_u32(tiles) + (uint32_t)kb * stage_bytes, full, l2_policy_evict_first());
    }
  }
  // TMEM only now: the blocks that an early one waits for may still have to allocate theirs
  if (early) qb_follow();
  if (warp == 1) {      // one warp allocates the accumulator columns (in a pair: the same warp of both blocks)
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                   ::"r"(smem_u32(&sh.tmem_base)), "r"((uint32_t)tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                   ::"r"(smem_u32(&sh.tmem_base)), "r"((uint32_t)tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if (MODE != 2 && gather_k > 0) {
    // the token rows are fetched one by one from the step's activations: row i of the tile is the token
    // of the i-th pair of this expert
    for (int i = threadIdx.x; i < rows; i += blockDim.x) s_pair[i] = sorted_pair[row0 + i] / gather_k;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();      // both blocks' barriers exist before either counts on the other's
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer: lane 0 waits and fetches the boxes; where the token rows are fetched
    // one by one, all lanes take their share of them ----------------
    // weights are read once per step by tiles of few rows (evict first); the 256-row tiles of one expert run at
    // about the same time and read the same weights, so those stay (measured: 5 % on a 16,384-token step)
    const uint64_t pol_w = PAIR ? l2_policy_evict_last() : l2_policy_evict_first(), pol_x = l2_policy_evict_last();
    const bool by_row = MODE != 2 && gather_k > 0;
    // tiles of more rows: four rows an instruction (the last valid row again where a group has fewer)
    const bool by_four = by_row && KS == 1 && NT > EG_FOUR_ROWS;
    // the tile rows this block fetches: all of them, or a pair's half
    const int r_lo = PAIR ? (int)rank * (n_mma / 2) : 0;
    const int r_hi = PAIR ? min(rows, r_lo + n_mma / 2) : rows;
    int armed = 0;
    // Nothing in this loop waits for memory, and it has to come round faster than the tensor cores use a stage (512 cycles for a pair's
    // two matrices): stage and parity are counted, addresses step, and lane 0 runs alone unless rows are fetched one by one.  With a
    // division by the number of stages a turn took 880 cycles, with rows one by one 1,140.
    auto fours = [](int n) { return n > 0 ? (n + 3) & ~3 : 0; };
    const int first_rows = PAIR ? min(rows, n_mma / 2) : rows;
    const uint32_t x_bytes = by_four ? (uint32_t)(fours(first_rows) + fours(rows - first_rows)) * BK * 2
                             : by_row ? (uint32_t)rows * BK * 2 : (PAIR ? 2u : 1u) * b_bytes;
    const uint32_t tx = (PAIR ? 2u : 1u) * NM * a_bytes + x_bytes;
    const uint32_t full0 = smem_u32(&sh.full[0]), empty0 = smem_u32(&sh.empty[0]), ring = smem_u32(tiles);
    // a pair: every copy of either block counts on the first block's barrier, which expects both blocks'
    // bytes (the second block's copies may count before the first has said so)
    const uint32_t bars = PAIR ? mapa_u32(full0, 0u) : full0;
    uint32_t st = ring, parity = 1u;
    int s = 0;
    auto turn = [&](int kb, bool weights) {      // lane 0: the boxes of a stage
      const uint32_t bar = bars + 8u * s;
      if (weights) {
        if (rank == 0) mbar_expect_tx(full0 + 8u * s, tx);
        load_weights(kb, st, bar, pol_w);
      }
      if (!by_row) {
        if constexpr (PAIR) tma_load_2d_pair(st + NM * a_bytes, &tm_x, kb * EG_BK, row0 + r_lo, bar, pol_x);
        else if constexpr (KS == 2) tma_load_3d(st + NM * a_bytes, &tm_x, 0, row0, kb * KS, bar, pol_x);
        else tma_load_2d(st + NM * a_bytes, &tm_x, kb * EG_BK, row0, bar, pol_x);
      }
    };
    auto next = [&] {
      st += stage_bytes;
      if (++s == stages) { s = 0; st = ring; parity ^= 1u; }
    };
    if (!by_row) {
      if (lane == 0) {
#pragma unroll 1
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(empty0 + 8u * s, parity, abort_flag)) break;
          turn(kb, kb >= ahead);      // an early block's first weights are on their way
          armed = kb + 1;
          next();
        }
      }
    } else {
#pragma unroll 1
      for (int kb = 0; kb < k_blocks; ++kb) {
        int ok = 1;
        if (lane == 0) ok = mbar_wait(empty0 + 8u * s, parity, abort_flag) ? 1 : 0;
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        if (lane == 0) turn(kb, true);
        // boxes of one row: the swizzle follows the shared-memory address, so a row lands where a box of
        // many rows would have put it; the rows past the expert's last keep what the stage held before, and
        // their columns of the product are never read
        if (by_four) {
          for (int i = r_lo + 4 * lane; i < r_hi; i += 128) {
            const int row[4] = {s_pair[i], s_pair[min(i + 1, r_hi - 1)], s_pair[min(i + 2, r_hi - 1)], s_pair[min(i + 3, r_hi - 1)]};
            const uint32_t dst = st + NM * a_bytes + (i - r_lo) * (EG_BK * 2);
            if (PAIR) tma_gather4_pair(dst, &tm_x, kb * BK, row, bars + 8u * s, pol_x);
            else tma_gather4(dst, &tm_x, kb * BK, row, bars + 8u * s, pol_x);
          }
        } else for (int i = r_lo + lane; i < r_hi; i += 32) {
          const uint32_t dst = st + NM * a_bytes + (i - r_lo) * (EG_BK * 2);
          if (PAIR) tma_load_2d_pair(dst, &tm_x, kb * BK, s_pair[i], bars + 8u * s, pol_x);
          else tma_load_2d(dst, &tm_x, kb * BK, s_pair[i], bars + 8u * s, pol_x);
          if (KS == 2) tma_load_2d(dst + b_slab, &tm_x, kb * BK + EG_BK, s_pair[i], bars + 8u * s, pol_x);      // zeros past the last slab
        }
        armed = kb + 1;
        next();
      }
    }
    if (lane == 0) {
      if (*abort_flag && PAIR && rank != 0) {
        // this block's copies count on the other block's barriers, which it cannot wait on: give them time
        const uint64_t t0 = global_ns();
        for (uint32_t it = 0; it < TC_SPIN_LIMIT && global_ns() - t0 < 100000ull; ++it) __nanosleep(1000);
      } else if (*abort_flag) {
        // let the copies that were issued land before this block's shared memory is given away
        for (int kb = max(0, armed - stages); kb < armed; ++kb) {
          const int s = kb % stages;
          const uint32_t ph = (uint32_t)(kb / stages) & 1u;
          const uint64_t t0 = global_ns();
          for (uint32_t it = 0; it < TC_SPIN_LIMIT && !mbar_try_wait(smem_u32(&sh.full[s]), ph); ++it)
            if ((it & 63u) == 63u && global_ns() - t0 > TC_WAIT_NS) break;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = umma_idesc(PAIR ? 2 * EG_M : EG_M, n_mma);
      bool ok = true;
      const uint32_t full0 = smem_u32(&sh.full[0]), empty0 = smem_u32(&sh.empty[0]);
      // the descriptors of the first stage's tiles; the address field counts 16 bytes
      const uint64_t a_first = umma_desc_sw128(smem_u32(tiles)), b_first = umma_desc_sw128(smem_u32(tiles) + NM * a_bytes);
      uint64_t at = 0;
      uint32_t parity = 0u, acc = 0u;
      int s = 0;
#pragma unroll 1
      for (int kb = 0; kb < k_blocks; ++kb) {
        ok = mbar_wait(full0 + 8u * s, parity, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int m = 0; m < NM; ++m) {
#pragma unroll
          for (int k16 = 0; k16 < BK / 16; ++k16) {
            // 16 k elements = 32 bytes further along the swizzled row: +2 in the 16-byte address field
            const int slab = k16 / (EG_BK / 16), in = k16 % (EG_BK / 16) * 2;
            const uint64_t a_desc = a_first + at + (uint64_t)((m * (int)a_bytes + slab * (int)A_SLAB) / 16 + in);
            const uint64_t b_desc = b_first + at + (uint64_t)(slab * (int)(b_slab >> 4) + in);
            if (PAIR) umma_bf16_pair(tmem_base + (uint32_t)(m * NT), a_desc, b_desc, idesc, k16 != 0 ? 1u : acc);
            else umma_bf16(tmem_base + (uint32_t)(m * NT), a_desc, b_desc, idesc, k16 != 0 ? 1u : acc);
          }
        }
        // the stage is free once these MMAs have read it
        if (PAIR) umma_commit_pair(empty0 + 8u * s); else umma_commit(empty0 + 8u * s);
        acc = 1u;
        at += stage_bytes >> 4;
        if (++s == stages) { s = 0; at = 0; parity ^= 1u; }
      }
      if (ok) {
        if (PAIR) umma_commit_pair(smem_u32(&sh.tmem_full)); else umma_commit(smem_u32(&sh.tmem_full));
      }
    }
  } else {
    // ---------------- epilogue: one TMEM lane quadrant a warp (a warp reaches the 32 lanes of its index
    // modulo 4); a pair's blocks have two warps a quadrant that take the column chunks in turn ----------------
    constexpr int SPLIT = PAIR ? 2 : 1;
    constexpr int EPI_THREADS = SPLIT * 128;
    const int quad = warp & 3, sub = (warp - 2) >> 2;
    float* ups = reinterpret_cast<float*>(tiles);      // HALF: [NT][64], over the ring when all products are done
    const int feat = j0 + quad * 32 + lane;
    if (MODE == 2 || (MODE == 1 && act.kind == 1)) {
      // where each row goes and its routing weight: fetched here, under the main loop, by the warps that
      // need them at its end (two dependent reads that the producer and the issuer do not wait for); no
      // weights: every row counts once
      for (int i = threadIdx.x - 64; i < NT; i += EPI_THREADS) {
        const int pr = i < rows ? sorted_pair[row0 + i] : 0;
        if (MODE == 2) s_pair[i] = pr;      // in the first product s_pair holds the token rows the producer fetches
        s_w[i] = i < rows ? (pair_w != nullptr ? pair_w[pr] : 1.f) : 0.f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");      // the epilogue warps
    }
    // tcgen05.ld / wait::ld are .sync.aligned: the whole warp runs them or none of it does, so the lanes
    // vote on the wait's answer (a lane may see another role's abort flag before its neighbour does)
    const bool acc_ready = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh.tmem_full), 0u, abort_flag) ? 1 : 0) != 0;
    if (acc_ready) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
      if (HALF && quad >= 2) {
        for (int c0 = 0; c0 < rows; c0 += 16) {
          uint32_t v[16];
          tmem_ld16(lane_addr + (uint32_t)c0, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 16; ++i) ups[(c0 + i) * (EG_M / 2) + (quad - 2) * 32 + lane] = __uint_as_float(v[i]);
        }
      }
    }
    if (HALF) asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
    if (acc_ready && !(HALF && quad >= 2)) {
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
      for (int c0 = 16 * sub; c0 < rows; c0 += 16 * SPLIT) {
        uint32_t v0[16], v1[16];
        tmem_ld16(lane_addr + (uint32_t)c0, v0);
        if (NM == 2) tmem_ld16(lane_addr + (uint32_t)(NT + c0), v1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // all 16 columns are computed (independent chains, one warp a scheduler has nothing else to hide
        // latency with); only the stores look at the row count
        if (MODE == 1) {
          __nv_bfloat16 r[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float g = __uint_as_float(v0[i]), u = HALF ? ups[(c0 + i) * (EG_M / 2) + quad * 32 + lane] : __uint_as_float(v1[i]);
            r[i] = __float2bfloat16_rn(act.kind == 1 ? clamped_glu(g, u, s_w[c0 + i], act) : silu_mul(g, u));
          }
          if (feat < N_out) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out) + (size_t)(row0 + c0) * N_out + feat;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c0 + i < rows) dst[(size_t)i * N_out] = r[i];
          }
        } else if (MODE == 3) {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out) + (size_t)(row0 + c0) * N_out;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (c0 + i < rows) {
              const float a = fmaxf(__uint_as_float(v0[i]), 0.f);
              if (feat < N_out) dst[(size_t)i * N_out + feat] = __float2bfloat16_rn(a * a);
              if (NM == 2 && feat + EG_M < N_out) {
                const float b = fmaxf(__uint_as_float(v1[i]), 0.f);
                dst[(size_t)i * N_out + feat + EG_M] = __float2bfloat16_rn(b * b);
              }
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int col = c0 + i;
            if (col < rows) {
              float* dst = reinterpret_cast<float*>(out) + (size_t)s_pair[col] * N_out;
              const float w = s_w[col];
              if (feat < N_out) dst[feat] = w * __uint_as_float(v0[i]);
              if (NM == 2 && feat + EG_M < N_out) dst[feat + EG_M] = w * __uint_as_float(v1[i]);
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // neither block of a pair leaves, or gives its accumulators back, while the other's MMAs may read its
  // shared memory or its epilogue its TMEM
  if (PAIR) cluster_sync_all();
  if (warp == 1) {
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)tmem_cols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)tmem_cols) : "memory");
  }
  if (threadIdx.x == 0 && sh.abort_flag) qb_set_status(status, QB_STATUS_WAIT_TIMEOUT, tile, 5);
}

#define QB_EG_PARAMS                                                                                              \
  const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, void* __restrict__ out,     \
      const int* sorted_pair, const float* pair_w, const int* plan, const int* tile_expert, const int* tile_row0, \
      int E, int K, int N_out, int NT, int stages, int tmem_cols, int gather_k, int* status, EgAct act, int early
#define QB_EG_ARGS tm_w, tm_x, out, sorted_pair, pair_w, plan, tile_expert, tile_row0, E, K, N_out, NT, stages, tmem_cols, gather_k, status, act, early

template <int MODE, int NM, int KS>
__global__ void __launch_bounds__(EG_THREADS, 2) expert_gemm_tc_kernel(QB_EG_PARAMS) {
  expert_gemm_tc_body<MODE, NM, false, KS>(QB_EG_ARGS);
}
template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(EG_PAIR_THREADS, 1) expert_gemm_tc_pair_kernel(QB_EG_PARAMS) {
  expert_gemm_tc_body<MODE, 2, true, 1>(QB_EG_ARGS);
}

// out[p, :] = x[sorted_pair[p] / top_k, :]   (rows of 16-byte chunks).  A warp takes a row, eight chunks a lane on their way; what is
// written does not stay in L2, so that x, whose rows are read top_k times, does.
// Bound by the bytes written: 8 rows a token of 3,072, 2,048 tokens 28.7 -> 23.6 us, 12,800 (708 MB) 172 -> 156 (a thread a chunk before).
constexpr int GR_WARPS = 8, GR_AHEAD = 8;
__global__ void __launch_bounds__(GR_WARPS * 32) gather_rows_kernel(const uint4* __restrict__ x, uint4* __restrict__ out,
                                                                    const int* __restrict__ sorted_pair, int n_pairs, int top_k, int chunks) {
  const int lane = threadIdx.x & 31, p = blockIdx.x * GR_WARPS + (threadIdx.x >> 5);
  if (p >= n_pairs) return;
  const uint4* src = x + (size_t)(sorted_pair[p] / top_k) * chunks;
  uint4* dst = out + (size_t)p * chunks;
  for (int c0 = lane; c0 < chunks; c0 += 32 * GR_AHEAD) {
    uint4 v[GR_AHEAD];
#pragma unroll
    for (int i = 0; i < GR_AHEAD; ++i)
      if (c0 + 32 * i < chunks) v[i] = src[c0 + 32 * i];
#pragma unroll
    for (int i = 0; i < GR_AHEAD; ++i)
      if (c0 + 32 * i < chunks) __stcs(dst + c0 + 32 * i, v[i]);
  }
}

// [rows, K / 64, 64], boxes of two slabs: [2][box_rows][64] in shared memory (zeros past the last slab)
int map_slabs(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows) {
  const cuuint64_t dims[3] = {EG_BK, rows, K / EG_BK}, strides[2] = {K * 2, EG_BK * 2};
  const cuuint32_t box[3] = {EG_BK, box_rows, 2};
  return make_map(map, base, 3, dims, strides, box);
}
// [experts, gate / up, I, K / 64, 64], boxes [2 slabs][gate, up][64 features][64]
int map_gate_up(CUtensorMap* map, const void* base, uint64_t experts, uint64_t I, uint64_t K) {
  const cuuint64_t dims[5] = {EG_BK, I, 2, K / EG_BK, experts}, strides[4] = {K * 2, I * K * 2, EG_BK * 2, 2 * I * K * 2};
  const cuuint32_t box[5] = {EG_BK, EG_M / 2, 2, 2, 1};
  return make_map(map, base, 5, dims, strides, box);
}

}  // namespace

extern "C" int qb_gather_rows(const void* x, void* out, const int* sorted_pair, int n_pairs, int top_k, int K,
                              cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (K % 8) return QB_ERR_UNSUPPORTED;
  gather_rows_kernel<<<(n_pairs + GR_WARPS - 1) / GR_WARPS, GR_WARPS * 32, 0, stream>>>((const uint4*)x, (uint4*)out, sorted_pair, n_pairs,
                                                                                      top_k, K / 8);
  QB_LAUNCH_CHECK();
  return 0;
}

// x_rows: bf16 [n_pairs, K] in sorted order (mode 1: the gathered activations; mode 2: the act rows); or,
// mode 1 with gather_k > 0, the step's activations [n_rows, K] themselves: the kernel fetches the row of
// token sorted_pair[p] / gather_k for pair p (for steps of few rows an expert).
// weights: bf16 [weight_experts, (mode 1 ? 2 : 1) * N_out, K] (weight_experts 0: E; fewer than E when the plan's
// last experts have no weights and no tiles).  NT: token tile (16..256, a multiple of 16); the plan's
// tile list must have been made with the same NT.
extern "C" int qb_expert_gemm_tc(int mode, const void* x_rows, const void* weights, void* out, const int* sorted_pair,
                                 const float* pair_w, const int* plan, const int* tile_expert, const int* tile_row0,
                                 int max_tiles, int n_pairs, int E, int K, int N_out, int NT, int gather_k, int n_rows,
                                 int* status, int weight_experts, int act_kind, float act_limit, float act_alpha,
                                 int after_first, cudaStream_t stream) {
  if (max_tiles <= 0 || n_pairs <= 0) return 0;
  if (act_kind < 0 || act_kind > 1 || (act_kind == 1 && (mode != 1 || pair_w == nullptr))) return QB_ERR_BAD_ARG;
  const EgAct act{act_kind, act_limit, act_alpha};
  if (weight_experts <= 0 || weight_experts > E) weight_experts = E;
  if (K % 8 || K <= 0 || N_out <= 0 || NT < 16 || NT > 256 || NT % 16 || max_tiles > 65535) return QB_ERR_UNSUPPORTED;
  if (mode != 1 && mode != 2 && mode != 3) return QB_ERR_BAD_ARG;
  // weight tiles a block: gate and up (mode 1); two blocks of 128 features for the down product of 256-row
  // token tiles (see the kernel)
  int sms = 0;
  const int rc_sms = sm_count(sms);
  if (rc_sms) return rc_sms;
  // the gated first product of so few tiles that blocks of 128 features would leave SMs idle: blocks of 64, gate and up in one weight tile
  // (one token, 8 of 256 experts of 3,072 x 1,536: 96 blocks 33.0 us with one slab a stage, 192 blocks of half the size 28.4)
  const bool half = mode == 1 && NT <= 32 && (size_t)((N_out + EG_M - 1) / EG_M) * (size_t)max_tiles <= (size_t)sms;
  const int nm = half ? 1 : (mode == 1 || NT >= 128) ? 2 : 1;
  const int feats = half ? EG_M / 2 : mode == 1 ? EG_M : nm * EG_M;
  // tiles of 256 token rows (steps bound by the tensor cores) are taken by pairs of blocks, see the kernel
  const bool pair = NT == 256;
  if (((uintptr_t)x_rows | (uintptr_t)weights) & 15) return QB_ERR_BAD_ARG;
  // Two blocks share an SM (shared memory is the limit), so that one block's prologue and epilogue run
  // under the other's main loop; each gets a ring of about 105 KB.
  // a tile of 256 token rows has a block to itself on its SM (its two accumulators fill the TMEM)
  // and so has every block of a launch of no more blocks than there are SMs (a single token's step)
  int grid_x = (N_out + feats - 1) / feats;
  if (pair) grid_x = (grid_x + 1) & ~1;      // a pair's second block may lie past the last feature: it drops its columns
  const size_t blocks = (size_t)grid_x * (size_t)max_tiles;
  const bool alone = NT > 128 || blocks <= (size_t)sms;
  // Launches of at most two blocks an SM are bound by how fast a block's producer and issuer go round: stages of two slabs (one token of
  // an 8-expert layer 2,048 x 2,112, 18 MB: 16.1 + 12.6 us for its two products with one slab a stage, 10.9 + 10.7 with two).
  const int ks = nm == 1 && NT <= 32 && K % EG_BK == 0 && blocks <= 2 * (size_t)sms ? 2 : 1;
  const uint64_t w_experts = (uint64_t)weight_experts, rows_x = (uint64_t)(gather_k > 0 ? n_rows : n_pairs);
  if (gather_k < 0 || (gather_k > 0 && (mode == 2 || n_rows <= 0))) return QB_ERR_BAD_ARG;
  CUtensorMap tm_w, tm_x;
  int rc;
  if (ks == 2 && half) rc = map_gate_up(&tm_w, weights, w_experts, (uint64_t)N_out, (uint64_t)K);
  else if (ks == 2) rc = map_slabs(&tm_w, weights, w_experts * N_out, (uint64_t)K, EG_M);
  else rc = map_2d(&tm_w, weights, w_experts * (mode == 1 ? 2 : 1) * N_out, (uint64_t)K, half ? EG_M / 2 : EG_M);
  if (rc) return rc;
  if (gather_k > 0) rc = map_2d(&tm_x, x_rows, rows_x, (uint64_t)K, 1u);
  else if (ks == 2) rc = map_slabs(&tm_x, x_rows, rows_x, (uint64_t)K, (uint32_t)NT);
  else rc = map_2d(&tm_x, x_rows, rows_x, (uint64_t)K, (uint32_t)(pair ? NT / 2 : NT));
  if (rc) return rc;
  const size_t stage_bytes = (size_t)ks * EG_BK * 2 * ((size_t)nm * EG_M + (size_t)(pair ? NT / 2 : NT));
  // Token tiles of at most 32 rows (decode steps of a few tokens: short blocks, one expert's 128 features
  // each): three blocks an SM with rings of about 70 KB hide a block's prologue and epilogue better than
  // two with 105 KB (measured at 8 tokens: 154 + 80 us against 161 + 86 us for the two products of a layer).
  int stages = (int)((size_t)(alone ? 200 * 1024 : ks == 2 ? 109 * 1024 : 105 * 1024) / stage_bytes);
  if (blocks > 2 * (size_t)sms && NT <= 32 && 72000 / stage_bytes >= 2) stages = (int)(72000 / stage_bytes);    // three blocks an SM
  // the down product of 64-row tiles (steps of 33 to 64 tokens): four blocks an SM with two stages each
  // (measured at 64 tokens: 308 us against 330 us)
  if (!alone && mode == 2 && NT == 64 && 50000 / stage_bytes >= 2) stages = (int)(50000 / stage_bytes);
  if (stages > 8) stages = 8;
  const int k_blocks = (K + ks * EG_BK - 1) / (ks * EG_BK);
  if (stages > k_blocks) stages = k_blocks;
  if (stages < 2 && k_blocks >= 2) return QB_ERR_UNSUPPORTED;
  const size_t smem = stage_bytes * stages + 1024;
  int tmem_cols = 32;
  while (tmem_cols < nm * NT) tmem_cols *= 2;
  dim3 grid(grid_x, max_tiles);
  const int early = mode == 2 && !pair && after_first ? 1 : 0;
  cudaError_t err;
#define QB_EG(KERNEL_, GK, THREADS_)                                                                                       \
  do {                                                                                                             \
    err = cudaFuncSetAttribute(KERNEL_, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                  \
    if (err != cudaSuccess) return (int)err;                                                                       \
    qb_launch(KERNEL_, grid, THREADS_, smem, stream, tm_w, tm_x, out, sorted_pair, pair_w, plan, tile_expert, tile_row0, E, K, \
              N_out, NT, stages, tmem_cols, GK, status, act, early);                                               \
  } while (0)
  if (pair && mode == 1) QB_EG(expert_gemm_tc_pair_kernel<1>, gather_k, EG_PAIR_THREADS);
  else if (pair && mode == 3) QB_EG(expert_gemm_tc_pair_kernel<3>, gather_k, EG_PAIR_THREADS);
  else if (pair) QB_EG(expert_gemm_tc_pair_kernel<2>, 0, EG_PAIR_THREADS);
  else if (ks == 2 && mode == 1) QB_EG((expert_gemm_tc_kernel<1, 1, 2>), gather_k, EG_THREADS);
  else if (ks == 2 && mode == 3) QB_EG((expert_gemm_tc_kernel<3, 1, 2>), gather_k, EG_THREADS);
  else if (ks == 2) QB_EG((expert_gemm_tc_kernel<2, 1, 2>), 0, EG_THREADS);
  else if (half) QB_EG((expert_gemm_tc_kernel<1, 1, 1>), gather_k, EG_THREADS);
  else if (mode == 1) QB_EG((expert_gemm_tc_kernel<1, 2, 1>), gather_k, EG_THREADS);
  else if (mode == 3 && nm == 2) QB_EG((expert_gemm_tc_kernel<3, 2, 1>), gather_k, EG_THREADS);
  else if (mode == 3) QB_EG((expert_gemm_tc_kernel<3, 1, 1>), gather_k, EG_THREADS);
  else if (nm == 2) QB_EG((expert_gemm_tc_kernel<2, 2, 1>), 0, EG_THREADS);
  else QB_EG((expert_gemm_tc_kernel<2, 1, 1>), 0, EG_THREADS);
#undef QB_EG
  QB_LAUNCH_CHECK();
  return 0;
}
