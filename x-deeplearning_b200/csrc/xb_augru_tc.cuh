// Attention-gated GRU (AUGRU) of the DIEN-style model on the tensor cores (included by xb_rnn.cu).
//
// Every candidate of a request walks the SAME input sequence x[r] (the interest-extractor states) with its own
// attention scores, so for candidate n and step t
//   [r|u] = sigmoid(h Wg_h + (x_t Wg_x + bg)),  c = tanh((r*h) Wc_h + (x_t Wc_x + bc)),
//   u' = (1 - a[n,t]) u,  h' = u' h + (1 - u') c
// where the bracketed terms depend on the request and the step only. One CTA owns 128 candidates of one request
// and walks the T steps on chip: the two per-candidate products are tcgen05 MMAs (A = h, then r*h, as fp16 in
// tensor memory; the recurrent weights stay in shared memory), and the request-side terms enter the same MMAs
// through a selector slot of the A operand (a 1 in the slot of the current step against B rows that hold the
// precomputed x_t terms), exactly as the split attention engine feeds its per-step bias. The state h stays in
// fp32 registers; it is rounded to fp16 only as an MMA operand. Only the final state is written (the model reads
// nothing else), the input sequence is read once per CTA instead of once per candidate.
//
// What bounds it is the chain of a step: gate product, gates, candidate product, blend. The tanh units alone need 54
// paired instructions a row and step at H = 36 (864 cycles of a scheduler's SFU); the rest of a step is tensor-memory
// round trips and MMA latency. So three warpgroups share a tile, a third of the columns each (a row's columns are
// independent between the products): every scheduler then has three warps to fill the waits of one another, r*h goes
// out before the update gate is evaluated, and the update gate's SFU work hides the candidate product. H is a
// compile-time constant: a run-time H made the update gates a local-memory array. 128 tiles of 100 steps, H = 36: 115 us,
// 121 with a copy of the code per group, 382 with one warpgroup a tile.
//
// Cell semantics: VecAttGRUCell.call, xdl-algorithm-solution/DIEN/script/utils.py:178-207 (the reference ships no
// inference operator for it). Shapes: H padded to Hp = 8*ceil(H/8) must leave 4 or more spare slots (H = 36 does).
#pragma once

namespace xb {
namespace {

constexpr int AU_GROUPS = 3;              // worker warpgroups: one candidate row per thread, a third of the columns
constexpr int AU_WORKERS = AU_GROUPS * 128;
constexpr int AU_MMA_WARP = AU_GROUPS * 4;
constexpr int AU_THREADS = AU_WORKERS + 32;

struct AuGeom {
  int hp, nch, selpos, k, n1, n2, ngrp;   // k: MMA K (h, selector slots, zero chunk); n1 = pad16(2H), n2 = pad16(H)
  int blk1, blk2;                         // bytes of one 8-wide k chunk of B1 / B2
  int c_acc2, c_a1, c_a2, cols, tmem_cols;
  int o_b1, o_b2, o_att, o_x, total;      // shared memory
};

__host__ __device__ constexpr AuGeom au_geom(int H, int T) {
  AuGeom g{};
  g.hp = (H + 7) / 8 * 8;
  g.nch = g.hp / 8;
  g.selpos = H & 7;
  g.k = (g.hp + 15) / 16 * 16;                 // the chunk after the last h chunk, if any, is all zero
  g.n1 = (2 * H + 15) / 16 * 16;
  g.n2 = (H + 15) / 16 * 16;
  g.ngrp = (T + 3) / 4;
  g.blk1 = g.n1 * 16;
  g.blk2 = g.n2 * 16;
  g.c_acc2 = g.n1;
  g.c_a1 = g.n1 + g.n2;
  g.c_a2 = g.c_a1 + g.k / 2;
  g.cols = g.c_a2 + g.k / 2;
  g.tmem_cols = g.cols <= 32 ? 32 : g.cols <= 64 ? 64 : g.cols <= 128 ? 128 : g.cols <= 256 ? 256 : 512;
  // B operands: [weight chunks 0..nch-2][selector blocks 0..ngrp-1][zero block], ascending in k
  int off = 0;
  g.o_b1 = off; off += (g.nch - 1 + g.ngrp + 1) * g.blk1;
  g.o_b2 = off; off += (g.nch - 1 + g.ngrp + 1) * g.blk2;
  g.o_att = off; off += 128 * ((T + 7) / 8 * 8) * 2;     // attention scores of the tile, [128][Tp] fp16
  g.o_x = off; off += T * g.hp * 2;                      // input sequence of the request, fp16
  g.total = (off + 15) / 16 * 16;
  return g;
}

struct AuParams {
  const __half* x; const __half* att; __half* y;
  const __half *Wg, *bg, *Wc, *bc;
  int requests, n_cand, T, H, tiles_per_req;
  uint32_t idesc1, idesc2;
};

// byte offset of k chunk c (for selector group grp) inside a B operand whose chunk blocks are `blk` bytes
__device__ __forceinline__ int au_chunk_off(const AuGeom& g, int blk, int c, int grp) {
  if (c < g.nch - 1) return c * blk;
  if (c == g.nch - 1) return (g.nch - 1 + grp) * blk;
  return (g.nch - 1 + g.ngrp) * blk;
}

// N consecutive tensor-memory columns of this thread's lane
template <int N>
__device__ __forceinline__ void au_tmem_st(uint32_t at, const uint32_t* r) {
  using namespace umma;
  if constexpr (N >= 8) { tmem_st8(at, r); au_tmem_st<N - 8>(at + 8, r + 8); }
  else if constexpr (N >= 4) { tmem_st4(at, r[0], r[1], r[2], r[3]); au_tmem_st<N - 4>(at + 4, r + 4); }
  else if constexpr (N >= 2) { tmem_st2(at, r[0], r[1]); au_tmem_st<N - 2>(at + 2, r + 2); }
  else if constexpr (N == 1) tmem_st1(at, r[0]);
}

// The steps of one worker thread: candidate row `row` of the tile, columns [C0, C0 + 2 np) of the state. The groups run the
// same code with their own offsets (a copy each would not stay in the instruction cache that they share); the last group
// also writes the selector slots, which follow the state in the A operand.
template <int H>
__device__ __forceinline__ void au_worker(const AuParams& p, int grp, const __half* att_row, uint32_t lane_addr, __half* out, bool valid,
                                          uint64_t* a1_full, uint64_t* acc1_full, uint64_t* a2_full, uint64_t* acc2_full) {
  using namespace umma;
  constexpr AuGeom G = au_geom(H, 1);                       // tensor-memory columns do not depend on T
  constexpr int CPG = (H + 2 * AU_GROUPS - 1) / (2 * AU_GROUPS) * 2, NP = CPG / 2;
  constexpr bool EVEN = CPG * AU_GROUPS == H;               // every group has CPG columns
  const int C0 = min(grp * CPG, H), np = EVEN ? NP : min(CPG, H - C0) / 2;
  const bool last = grp == AU_GROUPS - 1;
  const int T = p.T, lane = threadIdx.x & 31;
  const uint32_t a1t = lane_addr + G.c_a1 + C0 / 2, a2t = lane_addr + G.c_a2 + C0 / 2;
  float h[CPG];
  uint32_t pk[NP], upk[NP];
#pragma unroll
  for (int i = 0; i < CPG; ++i) h[i] = 0.f;
#pragma unroll
  for (int i = 0; i < NP; ++i) pk[i] = upk[i] = 0u;
  auto publish = [&](uint32_t at, uint32_t operand, uint64_t* bar, int t) {
    if constexpr (EVEN) {
      au_tmem_st<NP>(at, pk);
    } else {
#pragma unroll
      for (int e = 0; e < NP; ++e)
        if (e < np) tmem_st1(at + e, pk[e]);
    }
    if (last) {
      const uint32_t one = (t & 1) ? 0x3C000000u : 0x3C00u;   // 1.0 in slot t % 4 of the four
      tmem_st2(operand + H / 2, (t & 2) ? 0u : one, (t & 2) ? one : 0u);
    }
    tmem_wait_st();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
  };
  if (last) {
    // what follows the selector slots (up to the operand's end) stays zero
    for (int c = H / 2 + 2; c < G.k / 2; ++c) { tmem_st1(lane_addr + G.c_a1 + c, 0u); tmem_st1(lane_addr + G.c_a2 + c, 0u); }
  }
  publish(a1t, lane_addr + G.c_a1, a1_full, 0);             // h_0 = 0 with the selector of step 0
  bool ok = true;
  // 16 or 32 columns in one load: more than the group's, still inside the allocation, the extra values are not used
  uint32_t vr[32], vu[32];
  auto load = [&](uint32_t at, uint32_t (&v)[32]) {
    if constexpr (CPG > 16) tmem_ld32_nowait(at, v);
    else tmem_ld16_lo_nowait(at, v);
  };
  auto loaded = [&](uint32_t (&v)[32]) {
    if constexpr (CPG > 16) tmem_wait_ld(v);
    else tmem_wait_ld(*reinterpret_cast<uint32_t(*)[16]>(&v));
  };
  // sigmoid(z) = 1/2 + 1/2 tanh(z/2), two columns per SFU instruction
  auto sigm2 = [](uint32_t a, uint32_t b) {
    const __half2 z = __floats2half2_rn(0.5f * __uint_as_float(a), 0.5f * __uint_as_float(b));
    const __half2 th = bits_h2(tanh_f16x2(h2_bits(z)));
    return __hfma2(th, __floats2half2_rn(0.5f, 0.5f), __floats2half2_rn(0.5f, 0.5f));
  };
  for (int t = 0; t < T; ++t) {
    const uint32_t ph = (uint32_t)t & 1u;
    // ---- gates: [r|u] = sigmoid(acc1); r*h becomes the A operand of the candidate product
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(acc1_full), ph, 32));
    if (!ok) break;
    tc_fence_after_sync();
    load(lane_addr + C0, vr);
    load(lane_addr + H + C0, vu);
    loaded(vr);
    loaded(vu);
#pragma unroll
    for (int e = 0; e < NP; ++e) {
      if (e < np) {
        const float2 rf = __half22float2(sigm2(vr[2 * e], vr[2 * e + 1]));
        pk[e] = h2_bits(__floats2half2_rn(rf.x * h[2 * e], rf.y * h[2 * e + 1]));
      }
    }
    publish(a2t, lane_addr + G.c_a2, a2_full, t);
#pragma unroll
    for (int e = 0; e < NP; ++e)
      if (e < np) upk[e] = h2_bits(sigm2(vu[2 * e], vu[2 * e + 1]));
    // ---- candidate and blend
    const float a = __half2float(att_row[t]);
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(acc2_full), ph, 33));
    if (!ok) break;
    tc_fence_after_sync();
    load(lane_addr + G.c_acc2 + C0, vr);
    loaded(vr);
#pragma unroll
    for (int e = 0; e < NP; ++e) {
      if (e < np) {
        const __half2 z = __floats2half2_rn(__uint_as_float(vr[2 * e]), __uint_as_float(vr[2 * e + 1]));
        const float2 c = __half22float2(bits_h2(tanh_f16x2(h2_bits(z))));
        const float2 u = __half22float2(bits_h2(upk[e]));
        const float u0 = (1.f - a) * u.x, u1 = (1.f - a) * u.y;
        h[2 * e] = u0 * h[2 * e] + (1.f - u0) * c.x;
        h[2 * e + 1] = u1 * h[2 * e + 1] + (1.f - u1) * c.y;
        pk[e] = h2_bits(__floats2half2_rn(h[2 * e], h[2 * e + 1]));
      }
    }
    if (t + 1 < T) publish(a1t, lane_addr + G.c_a1, a1_full, t + 1);
  }
  if (ok && valid) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (i < np) *reinterpret_cast<uint32_t*>(out + C0 + 2 * i) = pk[i];      // H is even: 4-byte aligned
  }
}

template <int H>
__global__ void __launch_bounds__(AU_THREADS, H <= 40 ? 2 : 1) augru_tc_kernel(const __grid_constant__ AuParams p) {
  using namespace umma;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[4];
  __shared__ uint32_t tmem_base_s;
  const AuGeom G = au_geom(H, p.T);
  constexpr AuGeom G1 = au_geom(H, 1);
  constexpr int hp = G1.hp, nch = G1.nch;
  const int T = p.T, tpp = (T + 7) / 8 * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x / p.tiles_per_req, tile = blockIdx.x % p.tiles_per_req;
  const int rows = min(128, p.n_cand - tile * 128);
  uint8_t* b1s = smem + G.o_b1;
  uint8_t* b2s = smem + G.o_b2;
  __half* atts = reinterpret_cast<__half*>(smem + G.o_att);
  __half* xs = reinterpret_cast<__half*>(smem + G.o_x);
  const __half zero = __float2half(0.f);
  pdl_wait();

  // ---- prologue -------------------------------------------------------------------------------------------
  // attention scores of the tile and the request's input sequence: asynchronous copies where alignment allows
  const __half* att_tile = p.att + ((int64_t)r * p.n_cand + tile * 128) * T;
  const bool a8 = (T % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.att) & 7) == 0);
  if (a8) {
    for (int idx = threadIdx.x; idx < rows * (T / 4); idx += AU_THREADS) {
      const int row = idx / (T / 4), pc = idx - row * (T / 4);
      cp_async8(atts + row * tpp + pc * 4, att_tile + (int64_t)row * T + pc * 4);
    }
  } else {
    for (int idx = threadIdx.x; idx < rows * T; idx += AU_THREADS) atts[(idx / T) * tpp + idx % T] = att_tile[idx];
  }
  const __half* xr = p.x + (int64_t)r * T * H;
  for (int idx = threadIdx.x; idx < T * hp; idx += AU_THREADS) {
    const int t = idx / hp, i = idx - t * hp;
    xs[idx] = i < H ? xr[t * H + i] : zero;
  }
  cp_async_commit();
  // recurrent weights as MMA B operands (row n = output column, k = index into h): chunk-major 8 x 16-byte blocks;
  // the last h chunk shares its block with the selector slots and is replicated into every selector block
  for (int idx = threadIdx.x; idx < G1.n1 * hp; idx += AU_THREADS) {
    const int i = idx / G1.n1, n = idx - i * G1.n1;
    const __half v = (n < 2 * H && i < H) ? p.Wg[(int64_t)(H + i) * 2 * H + n] : zero;
    const int c = i >> 3, e = i & 7;
    if (c < nch - 1) reinterpret_cast<__half*>(b1s + c * G1.blk1)[n * 8 + e] = v;
    else for (int g = 0; g < G.ngrp; ++g) reinterpret_cast<__half*>(b1s + (nch - 1 + g) * G1.blk1)[n * 8 + e] = v;
  }
  for (int idx = threadIdx.x; idx < G1.n2 * hp; idx += AU_THREADS) {
    const int i = idx / G1.n2, n = idx - i * G1.n2;
    const __half v = (n < H && i < H) ? p.Wc[(int64_t)(H + i) * H + n] : zero;
    const int c = i >> 3, e = i & 7;
    if (c < nch - 1) reinterpret_cast<__half*>(b2s + c * G1.blk2)[n * 8 + e] = v;
    else for (int g = 0; g < G.ngrp; ++g) reinterpret_cast<__half*>(b2s + (nch - 1 + g) * G1.blk2)[n * 8 + e] = v;
  }
  for (int i = threadIdx.x; i < G1.blk1 / 16; i += AU_THREADS)
    reinterpret_cast<uint4*>(b1s + (nch - 1 + G.ngrp) * G1.blk1)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < G1.blk2 / 16; i += AU_THREADS)
    reinterpret_cast<uint4*>(b2s + (nch - 1 + G.ngrp) * G1.blk2)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();                       // xs and the weight blocks are in place
  // request-side terms into the selector slots: slot t % 4 of selector block t / 4 holds, for output column n,
  //   B1: x_t Wg_x[:, n] + bg[n]      B2: x_t Wc_x[:, n] + bc[n]     (fp32 sums, rounded once)
  // A thread keeps one weight column in registers and takes every AU_GROUPS-th step.
  if (threadIdx.x < AU_WORKERS) {
    for (int nn = threadIdx.x & 127; nn < G1.n1 + G1.n2; nn += 128) {
      const bool first = nn < G1.n1;
      const int n = first ? nn : nn - G1.n1;
      const int width = first ? 2 * H : H;
      const bool in = n < width;
      const __half* W = first ? p.Wg : p.Wc;
      uint8_t* blks = first ? b1s + (nch - 1) * G1.blk1 : b2s + (nch - 1) * G1.blk2;
      const int blk = first ? G1.blk1 : G1.blk2;
      float w[H];
#pragma unroll
      for (int i = 0; i < H; ++i) w[i] = in ? __half2float(__ldg(W + i * width + n)) : 0.f;
      const float bias = in ? __half2float(first ? p.bg[n] : p.bc[n]) : 0.f;
      for (int t = threadIdx.x >> 7; t < G.ngrp * 4; t += AU_GROUPS) {
        float v = 0.f;
        if (t < T) {
          v = bias;
#pragma unroll
          for (int i = 0; i < H; i += 2) {
            const float2 xv = __half22float2(*reinterpret_cast<const __half2*>(xs + t * hp + i));
            v = fmaf(xv.x, w[i], v);
            v = fmaf(xv.y, w[i + 1], v);
          }
        }
        reinterpret_cast<__half*>(blks + (t >> 2) * blk)[n * 8 + G1.selpos + (t & 3)] = __float2half_rn(v);
      }
    }
  }
  // barriers: a1_full (every worker warp: h operand of a step written), acc1_full (gate product done),
  //           a2_full (every worker warp: r*h written), acc2_full (candidate product done)
  uint64_t* a1_full = &bars[0];
  uint64_t* acc1_full = &bars[1];
  uint64_t* a2_full = &bars[2];
  uint64_t* acc2_full = &bars[3];
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(a1_full), AU_WORKERS / 32);
    mbar_init(smem_u32(acc1_full), 1);
    mbar_init(smem_u32(a2_full), AU_WORKERS / 32);
    mbar_init(smem_u32(acc2_full), 1);
    fence_barrier_init();
  }
  if (warp == AU_MMA_WARP) tmem_alloc(smem_u32(&tmem_base_s), (uint32_t)G1.tmem_cols);
  cp_async_wait_all();
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem0 = tmem_base_s;

  if (warp == AU_MMA_WARP) {
    // whole warp in uniform control flow, one elected lane issues: the descriptors stay in uniform registers
    {
      constexpr int nks = G1.k / 16, sel_ks = (nch - 1) / 2;            // nks <= 4 (H <= 64)
      const uint32_t b1a = smem_u32(b1s), b2a = smem_u32(b2s);
      // descriptors for selector group 0; only the k step with the selector chunk moves with the group
      uint64_t d1[4], d2[4], delta1 = 0, delta2 = 0;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        d1[ks] = d2[ks] = 0;
        if (ks < nks) {
          const uint32_t o0 = au_chunk_off(G, G1.blk1, 2 * ks, 0), o1 = au_chunk_off(G, G1.blk1, 2 * ks + 1, 0);
          const uint32_t q0 = au_chunk_off(G, G1.blk2, 2 * ks, 0), q1 = au_chunk_off(G, G1.blk2, 2 * ks + 1, 0);
          d1[ks] = make_desc_interleaved(b1a + o0, o1 - o0, 128);
          d2[ks] = make_desc_interleaved(b2a + q0, q1 - q0, 128);
          if (ks == sel_ks && G.ngrp > 1) {
            const uint32_t r0 = au_chunk_off(G, G1.blk1, 2 * ks, 1), r1 = au_chunk_off(G, G1.blk1, 2 * ks + 1, 1);
            const uint32_t s0 = au_chunk_off(G, G1.blk2, 2 * ks, 1), s1 = au_chunk_off(G, G1.blk2, 2 * ks + 1, 1);
            delta1 = make_desc_interleaved(b1a + r0, r1 - r0, 128) - d1[ks];
            delta2 = make_desc_interleaved(b2a + s0, s1 - s0, 128) - d2[ks];
          }
        }
      }
      for (int t = 0; t < T; ++t) {
        const uint32_t ph = (uint32_t)t & 1u;
        const uint64_t grp = (uint64_t)(t >> 2);
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(a1_full), ph, 30))) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          if (ks < nks)
            mma_f16_ts_elect(tmem0, tmem0 + G1.c_a1 + 8 * ks, d1[ks] + (ks == sel_ks ? grp * delta1 : 0ull), p.idesc1, ks > 0 ? 1u : 0u);
        mma_commit_elect(smem_u32(acc1_full));
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(a2_full), ph, 31))) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          if (ks < nks)
            mma_f16_ts_elect(tmem0 + G1.c_acc2, tmem0 + G1.c_a2 + 8 * ks, d2[ks] + (ks == sel_ks ? grp * delta2 : 0ull), p.idesc2,
                             ks > 0 ? 1u : 0u);
        mma_commit_elect(smem_u32(acc2_full));
      }
    }
  } else {
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = tmem0 + ((uint32_t)((warp & 3) * 32) << 16);
    const __half* att_row = atts + row * tpp;
    __half* out = p.y + ((int64_t)r * p.n_cand + tile * 128 + row) * H;
    au_worker<H>(p, warp >> 2, att_row, lane_addr, out, row < rows, a1_full, acc1_full, a2_full, acc2_full);
  }
  pdl_release();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == AU_MMA_WARP) {
    tc_fence_after_sync();
    tmem_dealloc(tmem0, (uint32_t)G1.tmem_cols);
  }
}

bool augru_tc_eligible(int H, int T) {
  if (H < 4 || H > 64 || (H & 1)) return false;
  const AuGeom g = au_geom(H, T);
  if (g.hp - H < 4) return false;                     // selector slots live in the padding of the last h chunk
  if (g.cols > 512 || g.n1 > 256) return false;
  return g.total <= 200 * 1024 && T >= 1;
}

template <int H>
int launch_augru_tc_h(const AuParams& p, unsigned blocks, int smem, cudaStream_t stream) {
  static PerDeviceOnce attr;                          // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr, 200 * 1024, (const void*)augru_tc_kernel<H>);
  launch_dependent(augru_tc_kernel<H>, blocks, AU_THREADS, smem, stream, p);
  return check_launch("augru_tc_kernel");
}

int launch_augru_tc(const AuParams& p0, cudaStream_t stream) {
  AuParams p = p0;
  const AuGeom g = au_geom(p.H, p.T);
  p.tiles_per_req = (p.n_cand + 127) / 128;
  p.idesc1 = umma::make_idesc(128, g.n1, 0);
  p.idesc2 = umma::make_idesc(128, g.n2, 0);
  const int64_t blocks = (int64_t)p.requests * p.tiles_per_req;
  XB_REQUIRE(blocks < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_augru_shared: too many tiles");
  // one instantiation per eligible H
  switch (p.H) {
#define XB_AU_CASE(h) case h: return launch_augru_tc_h<h>(p, (unsigned)blocks, g.total, stream)
    XB_AU_CASE(4); XB_AU_CASE(10); XB_AU_CASE(12); XB_AU_CASE(18); XB_AU_CASE(20); XB_AU_CASE(26); XB_AU_CASE(28);
    XB_AU_CASE(34); XB_AU_CASE(36); XB_AU_CASE(42); XB_AU_CASE(44); XB_AU_CASE(50); XB_AU_CASE(52); XB_AU_CASE(58);
    XB_AU_CASE(60);
#undef XB_AU_CASE
    default: return fail(XB_ERR_UNSUPPORTED, "xb_augru_shared: H = %d", p.H);
  }
}

}  // namespace
}  // namespace xb
