// Two-CTA form of the tcgen05 GEMM engine (included by xb_gemm_umma.cu): a cluster of two CTAs computes one
// 256 x 256 output tile with cta_group::2 MMAs, for large products with both operands K-major.
//
// What bounds the one-CTA form on such a product is the operand stream: a 128 x 256 tile takes 48 KB of shared
// memory per 64-deep k block, so three ring stages fill the SM and cover about a thousand cycles of L2 latency, and
// the MMAs read 12 KB per 128 cycles on top of the 48 KB per 512 that the loads write. A pair shares the B tile: each
// CTA loads its own 128 rows of A and half of the 256 rows of B (32 KB a block, five stages), and the leader's MMA reads
// both halves. Each CTA keeps the accumulator of its own 128 rows in its tensor memory, so the epilogue is that of the
// one-CTA kernel. Each CTA loads what it needs itself; nothing is multicast but the arrivals of tcgen05.commit.
// [65536, 1280] x [1280, 1024] bf16 + bias + PReLU and the 1024-512-256 layers after it: 207 us, 290 with one CTA a tile.
// Results leave by TMA (two-byte ones), which the epilogue of a layer with K <= 640 waited for: those three layers and the last one
// 226 -> 219 us, 640-512-256-1 on 65536 rows 81 -> 74, [65536, 256] x [256, 256] 22.4 -> 19.3. One staging area a warp: a second costs
// a stage of the ring (235, 78 and 19.9 us).
#pragma once

namespace xb {
namespace {

constexpr int PAIR_N = 256;                         // columns of a tile; rows: 128 per CTA
constexpr int PAIR_B_BYTES = (PAIR_N / 2) * BLOCK_K * 2;
constexpr int PAIR_STAGE_BYTES = A_STAGE_BYTES + PAIR_B_BYTES;
constexpr int PAIR_MAX_STAGES = 6;
constexpr int PAIR_Y_BUFS = 1;                      // staging areas of an epilogue warp

// TMA tile load into this CTA that signals a barrier of the pair's leader
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void mma_f16_ss_pair_elect(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at this address in both CTAs once every MMA issued so far has completed
__device__ __forceinline__ void mma_commit_pair_elect(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}

template <typename TOut>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_umma_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_y,
                      const __grid_constant__ UmmaGemmParams p) {
  using namespace umma;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int STAGES = p.stages;
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * A_STAGE_BYTES;
  __shared__ __align__(8) uint64_t full_bar[PAIR_MAX_STAGES];      // used in the leader: operands of both CTAs have landed
  __shared__ __align__(8) uint64_t empty_bar[PAIR_MAX_STAGES];     // in each CTA: the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_full[2];                    // in each CTA: accumulator complete
  __shared__ __align__(8) uint64_t acc_empty[2];                   // used in the leader: both CTAs' epilogues have drained it
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = blockIdx.x & 1;                           // 0: leader
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  // tiles_m counts 256-row tiles here; the n tiles of one row of tiles are neighbours in the sequence, so its A rows come
  // from HBM once and the pairs that work on it share them in L2
  const uint32_t total_tiles = (uint32_t)p.tiles_m * (uint32_t)p.tiles_n * (uint32_t)p.batch;
  const uint32_t tile_first = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  auto place = [&](uint32_t tile, int& b, int& m0, int& n0) {
    const uint32_t row = tile / (uint32_t)p.tiles_n;
    n0 = (int)(tile - row * (uint32_t)p.tiles_n) * PAIR_N;
    b = (int)(row / (uint32_t)p.tiles_m);
    m0 = (int)((row - (uint32_t)b * (uint32_t)p.tiles_m) * 2 + crank) * BLOCK_M;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&full_bar[s]), 1); mbar_init(smem_u32(&empty_bar[s]), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&acc_full[s]), 1); mbar_init(smem_u32(&acc_empty[s]), 2 * EPI_WARPS); }
    fence_barrier_init();
    if (sizeof(TOut) == 2) prefetch_tensormap(&map_y);
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
  }
  if (warp == 1) tmem_alloc_pair(smem_u32(&tmem_base_s), 2 * PAIR_N);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();                                                  // the other CTA's barriers are initialised too
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (uint32_t tile = tile_first; tile < total_tiles && ok; tile += tile_step) {
        int b, m0, n0;
        place(tile, b, m0, n0);
        for (int kb = 0; kb < num_kb; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
          ok = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, 41);
          if (!ok) break;
          // the leader expects the bytes of both CTAs; the other CTA's may arrive first, which the barrier allows (the
          // phase cannot complete before the leader's own arrival)
          if (crank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[s]), 2 * PAIR_STAGE_BYTES);
          const uint32_t bar = cluster_addr(smem_u32(&full_bar[s]), 0);
          tma_load_3d_pair(smem_u32(smem_a + s * A_STAGE_BYTES), &map_a, bar, kb * BLOCK_K, m0, p.a_batched ? b : 0);
          tma_load_3d_pair(smem_u32(smem_b + s * PAIR_B_BYTES), &map_b, bar, kb * BLOCK_K, n0 + (int)crank * (PAIR_N / 2), p.b_batched ? b : 0);
        }
      }
      // the leader's last arrivals have reached this CTA before it may leave (a stage that was never filled is free)
      for (int i = 0; i < STAGES && ok; ++i, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u))
        ok = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, 45);
    }
  } else if (warp == 1) {
    if (crank == 0) {
      int s = 0, it = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (uint32_t tile = tile_first; tile < total_tiles && ok; tile += tile_step, ++it) {
        const int as = it & 1;
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(smem_u32(&acc_empty[as]), ((uint32_t)(it >> 1) & 1u) ^ 1u, 44));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tmem_acc = tmem_base + as * PAIR_N;
        for (int kb = 0; kb < num_kb; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[s]), ph, 42));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(smem_a + s * A_STAGE_BYTES), b_addr = smem_u32(smem_b + s * PAIR_B_BYTES);
#pragma unroll
          for (int k = 0; k < BLOCK_K / 16; ++k)
            mma_f16_ss_pair_elect(tmem_acc, make_desc_sw128(a_addr + k * 32, 1024), make_desc_sw128(b_addr + k * 32, 1024), p.idesc,
                                  (kb > 0 || k > 0) ? 1u : 0u);
          mma_commit_pair_elect(smem_u32(&empty_bar[s]));
        }
        mma_commit_pair_elect(smem_u32(&acc_full[as]));
      }
    }
  } else {
    const int ew = warp - 2, q = warp & 3, part = ew >> 2, row = q * 32 + lane;
    [[maybe_unused]] const int c_begin = PAIR_N / 16 * part / 4, c_end = PAIR_N / 16 * (part + 1) / 4;
    float* s_bias = reinterpret_cast<float*>(smem + STAGES * PAIR_STAGE_BYTES);                    // [4][256]
    uint8_t* area = reinterpret_cast<uint8_t*>(s_bias + 4 * 256) + ew * PAIR_Y_BUFS * 32 * 64;
    uint32_t turn = 0;
    float *s_a = s_bias + 256, *s_b = s_a + 256, *s_c = s_b + 256;
    int it = 0, cur_n0 = -1, cur_b = -1;
    bool ok = true;
    // (a warp whose wait ran out keeps walking the tiles for the named barriers, as in the one-CTA kernel)
    for (uint32_t tile = tile_first; tile < total_tiles; tile += tile_step, ++it) {
      int b, m0, n0;
      place(tile, b, m0, n0);
      const int as = it & 1, gm = m0 + row;
      if (n0 != cur_n0 || b != cur_b) {
        cur_n0 = n0; cur_b = b;
        asm volatile("bar.sync 2, 512;" ::: "memory");
        const int e = ew * 32 + lane;
        if (e < PAIR_N) stage_columns(p, b, n0 + e, e, s_bias, s_a, s_b, s_c);
        asm volatile("bar.sync 2, 512;" ::: "memory");
      }
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[as]), (uint32_t)(it >> 1) & 1u, 43));
      if (!ok) continue;
      tc_fence_after_sync();
      const uint32_t tmem_acc = tmem_base + as * PAIR_N + ((uint32_t)(q * 32) << 16);
      const int y = m0 + q * 32, rows = p.M - y;                   // of the warp's 32; the columns are all there
      with_kind(p.epi.kind, [&](auto kind) {
        constexpr int KIND = decltype(kind)::value;
        if constexpr (sizeof(TOut) == 2)
          epi_tile_tma<TOut, KIND, 32>(map_y, tmem_acc, part, PAIR_N, p.alpha, s_bias, s_a, s_b, s_c, area, PAIR_Y_BUFS, turn, n0,
                                       p.y_beside ? b : y, p.y_beside ? y : b, rows > 0, lane);
        else
          epi_tile_fast<TOut, KIND>(tmem_acc, c_begin, c_end, p.alpha, s_bias, s_a, s_b, s_c,
                                    reinterpret_cast<TOut*>(p.Y) + (int64_t)b * p.stride_y + (int64_t)gm * p.ldy + n0, p.ldy, rows, PAIR_N, nullptr, lane);
      });
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(smem_u32(&acc_empty[as]), 0);
    }
    if (sizeof(TOut) == 2 && lane == 0) tma_store_wait_read<0>();
  }

  pdl_release();
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();                  // no CTA leaves while the other's MMAs, copies or arrivals may still touch it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 2 * PAIR_N);
  }
}

}  // namespace
}  // namespace xb
