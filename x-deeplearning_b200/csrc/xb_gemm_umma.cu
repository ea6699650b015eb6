// tcgen05 GEMM engine with fused bias + activation epilogue, and the xb_gemm
// dispatcher.
//
//   Y[b] = act(alpha * A[b] * B[b]^T + beta * bias[b])
//   A [M,K] row-major (K-major), B [N,K] row-major (K-major) or [K,N] row-major
//   (N-major, the layout Blaze holds weights in), fp16 or bf16, fp32 accumulation
//   in tensor memory.
//
// Persistent kernel, one CTA per SM, 128 x BLOCK_N output tiles. Warp 0 streams
// 128x64 A tiles (and BLOCK_Nx64 B tiles) through a shared-memory ring with TMA
// (as many stages as fit; 128-byte swizzle, out-of-range rows/columns zero-filled
// by the TMA unit, so M, N and K tails need no padding in HBM). When the whole
// B tile (all of K) is small and many m tiles share it, it is loaded once and stays
// resident while the CTA walks a contiguous run of tiles. Warp 1 issues
// tcgen05.mma (128 x BLOCK_N x 16 per instruction) into one of two TMEM
// accumulators and releases ring slots with tcgen05.commit. Warps 2-17 read the
// accumulator with tcgen05.ld (one output row per thread, a quarter of the
// columns per warpgroup), apply bias and activation and store with an arbitrary
// row stride, which is what lets parallel branches write side by side into one
// wide output (axis-1 concat) or stacked (axis 0).
#include <algorithm>
#include <mutex>
#include <cstring>
#include <type_traits>

#include "xb_common.cuh"
#include "xb_umma.cuh"

namespace xb {

int gemm_simt(const xb_gemm_args& a, cudaStream_t stream);
bool gemm_narrow_takes(const xb_gemm_args& a);           // (gemm_simt hands those to their own kernel)

namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;
constexpr int MAX_STAGES = 8;       // the launch picks as many as fit in shared memory (at least 2)
constexpr int SMEM_BUDGET = 220 * 1024;
constexpr int A_STAGE_BYTES = BLOCK_M * BLOCK_K * 2;
constexpr int MN_BOX_BYTES = 64 * BLOCK_K * 2;      // one N-major box: 64 k rows of 64 columns (128 bytes each)

struct UmmaGemmParams {
  int M, N, K, block_n, tmem_cols, tiles_m, tiles_n, batch, stages;
  int b_resident;        // the B tile (all of K) stays in shared memory while consecutive tiles share it
  int b_mn;              // B is [K,N] row-major: the MMA reads N-major tiles of 64 columns x 64 k
  int n_fast;            // consecutive tiles walk n first
  uint32_t tiles_per_cta;
  float alpha, beta;
  int a_batched, b_batched;
  const void* bias; int64_t ldbias, stride_bias; int bias_kind, bias_dtype, bias_group;
  void* Y; int64_t ldy, stride_y; int y_dtype;
  EpiParams epi; int64_t stride_ep;
  uint32_t idesc;
  int y_unit, y_bufs;    // results stored by TMA: columns of a copy (32 or 16), staging areas of a warp
  int y_beside;          // the batches lie beside one another in a row of Y: its map has the batch before the row
};

template <typename TOut>
__device__ __forceinline__ void store_row16(TOut* dst, const float (&v)[16], int valid, bool vec_ok) {
  if (sizeof(TOut) == 2 && vec_ok && valid == 16) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      TOut lo = from_f32<TOut>(v[2 * i]), hi = from_f32<TOut>(v[2 * i + 1]);
      w[i] = (uint32_t)(*reinterpret_cast<uint16_t*>(&lo)) | ((uint32_t)(*reinterpret_cast<uint16_t*>(&hi)) << 16);
    }
    uint4* d = reinterpret_cast<uint4*>(dst);
    d[0] = make_uint4(w[0], w[1], w[2], w[3]);
    d[1] = make_uint4(w[4], w[5], w[6], w[7]);
  } else if (sizeof(TOut) == 4 && vec_ok && valid == 16) {
    float4* d = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < valid) dst[i] = from_f32<TOut>(v[i]);
  }
}

// 16 epilogue warps: four per TMEM lane quarter, each owning a quarter of the tile's columns, so every
// scheduler has four of them to hide the TMEM round trip and the store latency behind one another
constexpr int EPI_WARPS = 16;
constexpr int GEMM_THREADS = 64 + EPI_WARPS * 32;

template <typename TOut>
__device__ __forceinline__ uint4 pack8(const float* v);
template <>
__device__ __forceinline__ uint4 pack8<__half>(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <>
__device__ __forceinline__ uint4 pack8<__nv_bfloat16>(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <>
__device__ __forceinline__ uint4 pack8<float>(const float*) { return make_uint4(0, 0, 0, 0); }   // not used

// 16 results of one output row as 16-byte stores, those that lie wholly in the `valid` columns left of it
template <typename TOut>
__device__ __forceinline__ void store16_vec(TOut* dst, const float (&v)[16], int valid) {
  if constexpr (sizeof(TOut) == 4) {
    float4* d = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (4 * i + 4 <= valid) d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
    uint4* d = reinterpret_cast<uint4*>(dst);
    if (8 <= valid) d[0] = pack8<TOut>(v);
    if (16 <= valid) d[1] = pack8<TOut>(v + 8);
  }
}

// Activation of 16 adjacent columns of one row; the per-column parameters sit in shared memory and are
// read as 16-byte vectors (all lanes read the same address: a broadcast).
template <int KIND>
__device__ __forceinline__ void epi_apply16(float (&v)[16], const float* s_a, const float* s_b, const float* s_c) {
  if constexpr (KIND != XB_EPI_NONE) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (KIND == XB_EPI_PRELU) {
      const float4 a = reinterpret_cast<const float4*>(s_a)[j];
      // x * (x < 0 ? w : 1): the same value as act_prelu for every x, signed zeros and NaN included
      v[4 * j] *= v[4 * j] < 0.f ? a.x : 1.f;
      v[4 * j + 1] *= v[4 * j + 1] < 0.f ? a.y : 1.f;
      v[4 * j + 2] *= v[4 * j + 2] < 0.f ? a.z : 1.f;
      v[4 * j + 3] *= v[4 * j + 3] < 0.f ? a.w : 1.f;
    } else if (KIND == XB_EPI_DICE) {
      const float4 g = reinterpret_cast<const float4*>(s_a)[j];
      const float4 b = reinterpret_cast<const float4*>(s_b)[j];
      const float4 c = reinterpret_cast<const float4*>(s_c)[j];
      const float gg[4] = {g.x, g.y, g.z, g.w}, bb[4] = {b.x, b.y, b.z, b.w}, cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float x = v[4 * j + i];
        const float pr = __fdividef(1.f, 1.f + __expf(-fmaf(x, cc[i], bb[i])));
        v[4 * j + i] = x * fmaf(pr, 1.f - gg[i], gg[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[4 * j + i] = act_sigmoid(v[4 * j + i]);
    }
  }
  }
}

constexpr int EPI_STAGE_BYTES = 32 * 64;      // per epilogue warp: 32 rows x 32 two-byte results

// Epilogue of a tile with a per-column bias (or none) and output rows of whole, aligned 16-byte pieces: this thread's row,
// columns [16 * c_begin, 16 * c_end) of the tile, as far as `rows` of the warp's 32 and `cols` of the tile's columns lie in the
// output (a piece is stored or it is not).
// Bound by shared memory's and L1's data path, which carries a result four times here (staging, both ways, beside the accumulator and
// the store). Ragged tiles went through epi_tile_edge before: [1000, 88] x [88, 168] fp16 4.8 us, 3.8 here; 8 x ([300, 256] x [256, 200])
// 5.1, 4.3.
// Two-byte outputs go through a 2 KB staging area of the warp: a thread holds 64 contiguous bytes of its
// own row, and a store instruction of one piece per lane would touch 32 different lines; after the
// exchange the 32 lanes of an instruction write 8 rows x 64 contiguous bytes. Piece j of row l is kept at
// position j ^ ((l >> 1) & 3) of the row, which makes both the writes (lane = row) and the reads (four
// lanes per row) free of bank conflicts.
template <typename TOut, int KIND, bool WHOLE = false>
__device__ __forceinline__ void epi_tile_fast(uint32_t tmem_row, int c_begin, int c_end, float alpha,
                                              const float* s_bias, const float* s_a, const float* s_b,
                                              const float* s_c, TOut* yrow, int64_t ldy, int rows, int cols,
                                              uint4* stage, int lane) {
  using namespace umma;
  for (int cg = c_begin; cg < c_end; cg += 2) {
    // two chunks per TMEM round trip when the thread owns two more
    uint32_t raw[32];
    const bool two = cg + 1 < c_end;                                    // uniform across the warp
    if (two) {
      tmem_ld32_nowait(tmem_row + (uint32_t)(cg * 16), raw);
    } else {
#pragma unroll
      for (int i = 16; i < 32; ++i) raw[i] = 0u;
      tmem_ld16_lo_nowait(tmem_row + (uint32_t)(cg * 16), raw);
    }
    tmem_wait_ld(raw);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !two) break;
      const int c = (cg + u) * 16;
      float v[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 b = reinterpret_cast<const float4*>(s_bias + c)[j];
        v[4 * j] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j]), b.x);
        v[4 * j + 1] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 1]), b.y);
        v[4 * j + 2] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 2]), b.z);
        v[4 * j + 3] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 3]), b.w);
      }
      epi_apply16<KIND>(v, s_a + c, s_b + c, s_c + c);
      if (sizeof(TOut) == 2 && two) {
        const int sw = (lane >> 1) & 3;
        stage[lane * 4 + ((2 * u) ^ sw)] = pack8<TOut>(v);
        stage[lane * 4 + ((2 * u + 1) ^ sw)] = pack8<TOut>(v + 8);
      } else if (WHOLE || lane < rows) {
        store16_vec<TOut>(yrow + c, v, WHOLE ? 16 : cols - c);
      }
    }
    if (sizeof(TOut) == 2 && two) {
      __syncwarp();
      const int slot = cg * 16 + (lane & 3) * 8;             // this lane's 16-byte column slot
      const int in = slot + 8 <= cols ? rows : 0;
      TOut* base = yrow + slot;                              // (in its own row)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        const uint4 x = stage[r * 4 + ((lane & 3) ^ ((r >> 1) & 3))];
        if (r < in) *reinterpret_cast<uint4*>(base + (int64_t)(r - lane) * ldy) = x;
      }
      __syncwarp();                                          // the next round overwrites the staging area
    }
  }
}

// A unit of W columns of this thread's row into the warp's staging area, as a W-column copy reads it (pieces swizzled as in
// epi_tile_fast; rows of 32 bytes where W = 16).
template <typename TOut, int KIND, int W>
__device__ __forceinline__ void epi_unit(uint32_t tmem_at, float alpha, const float* s_bias, const float* s_a, const float* s_b, const float* s_c,
                                         uint4* area, int lane) {
  using namespace umma;
  uint32_t raw[W];
  if constexpr (W == 32) tmem_ld32_nowait(tmem_at, raw);
  else tmem_ld16_nowait(tmem_at, raw);
  tmem_wait_ld(raw);
  const int sw = W == 32 ? (lane >> 1) & 3 : (lane >> 2) & 1;
#pragma unroll
  for (int u = 0; u < W / 16; ++u) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 b = reinterpret_cast<const float4*>(s_bias + 16 * u)[j];
      v[4 * j] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j]), b.x);
      v[4 * j + 1] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 1]), b.y);
      v[4 * j + 2] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 2]), b.z);
      v[4 * j + 3] = fmaf(alpha, __uint_as_float(raw[16 * u + 4 * j + 3]), b.w);
    }
    epi_apply16<KIND>(v, s_a + 16 * u, s_b + 16 * u, s_c + 16 * u);
    area[lane * (W / 8) + ((2 * u) ^ sw)] = pack8<TOut>(v);
    area[lane * (W / 8) + ((2 * u + 1) ^ sw)] = pack8<TOut>(v + 8);
  }
}

template <typename F>
__device__ __forceinline__ void with_kind(int kind, F f) {
  switch (kind) {
    case XB_EPI_PRELU: f(std::integral_constant<int, XB_EPI_PRELU>()); break;
    case XB_EPI_DICE: f(std::integral_constant<int, XB_EPI_DICE>()); break;
    case XB_EPI_SIGMOID: f(std::integral_constant<int, XB_EPI_SIGMOID>()); break;
    default: f(std::integral_constant<int, XB_EPI_NONE>()); break;
  }
}

// Epilogue of a tile whose results leave by TMA, a warp's 32 rows x W columns at a time: units `part`, `part` + 4, ... of the tile.
// A warp with two units a tile has two areas, so that it fills one while the other is read. What the threads' own stores and their
// reads of the staging area took of the data path (4900 wavefronts a tile of 128 x 256, 5000 cycles) is the copy engine's work here.
// [65536, 88] x [88, 256] fp16: 16.1 -> 11.8 us, N = 192 14.4 -> 10.5, 8 x ([4096, 256] x [256, 128]) side by side 8.3 -> 7.9.
// A sigmoid's division is most of an epilogue that has one (8 x ([33434, 88] x [88, 32]) 32 us, 20 without an activation).
// A turn is a copy: the wait counts committed groups, so a warp whose rows all lie past the output (`rows` false) takes no turn and
// leaves the areas as they are. (With turns that commit nothing, the wait for all but the latest copy would name the copy of the other
// area, and a later unit could overwrite what that copy still reads.)
template <typename TOut, int KIND, int W>
__device__ __forceinline__ void epi_tile_tma(const CUtensorMap& map_y, uint32_t tmem_row, int part, int cols, float alpha, const float* s_bias,
                                             const float* s_a, const float* s_b, const float* s_c, uint8_t* stage, int bufs, uint32_t& turn,
                                             int x, int y, int z, bool rows, int lane) {
  using namespace umma;
  if (!rows) return;                                         // (the same for the warp)
  for (int c = part * W; c < cols; c += 4 * W) {
    uint8_t* area = stage + (bufs == 2 ? (turn & 1u) * (32 * W * 2) : 0u);
    ++turn;
    if (lane == 0) {                                         // the copy that read this area last has done so
      if (bufs == 2) tma_store_wait_read<1>();
      else tma_store_wait_read<0>();
    }
    __syncwarp();
    epi_unit<TOut, KIND, W>(tmem_row + (uint32_t)c, alpha, s_bias + c, s_a + c, s_b + c, s_c + c, reinterpret_cast<uint4*>(area), lane);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) tma_store_3d(&map_y, smem_u32(area), x + c, y, z);
  }
}

// bias and activation parameters of output column gn into entry e of the staged columns
__device__ __forceinline__ void stage_columns(const UmmaGemmParams& p, int b, int gn, int e, float* s_bias, float* s_a, float* s_b,
                                              float* s_c) {
  const bool in = gn < p.N;
  float bv = 0.f, pa = 0.f, pb = 0.f, pc = 0.f;
  if (in && p.bias_kind == XB_BIAS_ROW) bv = p.beta * load_as_f32(p.bias, (int64_t)b * p.stride_bias + gn, p.bias_dtype);
  if (in && p.epi.kind == XB_EPI_PRELU) pa = p.epi.a[(int64_t)b * p.stride_ep + (p.epi.count == 1 ? 0 : gn)];
  if (in && p.epi.kind == XB_EPI_DICE) {
    const float var = p.epi.c[(int64_t)b * p.stride_ep + gn];
    pa = p.epi.a[(int64_t)b * p.stride_ep + gn];                            // gamma
    pc = p.epi.nosqrt ? 1.f / var : rsqrtf(var + 1e-8f);                    // 1/std
    pb = -p.epi.b[(int64_t)b * p.stride_ep + gn] * pc;                      // -mean/std
  }
  s_bias[e] = bv; s_a[e] = pa; s_b[e] = pb; s_c[e] = pc;
}

// Epilogue of any output: rows that start or end anywhere, a full bias matrix where there is one.
template <typename TOut>
__device__ __forceinline__ void epi_tile_edge(const UmmaGemmParams& p, uint32_t tmem_row, int c_begin, int c_end, const float* s_bias,
                                              const float* s_a, const float* s_b, const float* s_c, TOut* yrow, int b, int gm,
                                              int brow, int n0, bool vec_base, uint16_t* stage, int lane) {
  using namespace umma;
  for (int cg = c_begin; cg < c_end; ++cg) {
    uint32_t raw[16];
    tmem_ld16_nowait(tmem_row + (uint32_t)(cg * 16), raw);
    tmem_wait_ld(raw);
    const int c = cg * 16, gn0 = n0 + c, valid = min(p.N - gn0, 16);
    if (valid <= 0) continue;                                        // uniform across the warp
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = fmaf(p.alpha, __uint_as_float(raw[i]), s_bias[c + i]);
    if (p.bias_kind == XB_BIAS_FULL && gm < p.M) {
      const int64_t base = (int64_t)b * p.stride_bias + (int64_t)brow * p.ldbias + gn0;
      const float* bf = reinterpret_cast<const float*>(p.bias) + base;
      if (p.bias_dtype == XB_F32 && valid == 16 && (reinterpret_cast<uintptr_t>(bf) & 15) == 0) {
        // fp32 rows (the per-group partial product of a pruned GEMM): four 16-byte loads, mostly one
        // address per warp since consecutive output rows share the bias row
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(bf) + i);
          v[4 * i] += p.beta * t.x; v[4 * i + 1] += p.beta * t.y;
          v[4 * i + 2] += p.beta * t.z; v[4 * i + 3] += p.beta * t.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i < valid) v[i] += p.beta * load_as_f32(p.bias, base + i, p.bias_dtype);
      }
    }
    if (p.epi.kind == XB_EPI_PRELU) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = act_prelu(v[i], s_a[c + i]);
    } else if (p.epi.kind == XB_EPI_DICE) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float g = s_a[c + i];
        const float pr = __fdividef(1.f, 1.f + __expf(-fmaf(v[i], s_c[c + i], s_b[c + i])));
        v[i] = v[i] * fmaf(pr, 1.f - g, g);
      }
    } else if (p.epi.kind == XB_EPI_SIGMOID) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = act_sigmoid(v[i]);
    }
    const bool vec = vec_base && ((gn0 * sizeof(TOut)) % 16 == 0);
    if (sizeof(TOut) == 2 && !(vec && valid == 16)) {
      // Rows that start anywhere: a store of one element per lane and row touches 32 lines, so the warp turns its 32 x 16 results
      // and writes two rows at a time. [65536, 256] x [256, 255] fp16: 173 -> 29 us; [40594, 104] x [104, 41] 24 -> 8.3;
      // 8 x ([4198, 48] x [48, 398]) with a sigmoid 170 -> 36.
      const int piece = (lane >> 2) & 1;                              // (swapped in every other four rows: no bank conflicts)
      reinterpret_cast<uint4*>(stage)[lane * 2 + piece] = pack8<TOut>(v);
      reinterpret_cast<uint4*>(stage)[lane * 2 + (piece ^ 1)] = pack8<TOut>(v + 8);
      __syncwarp();
      const int col = lane & 15, rows = p.M - (gm - lane);            // (gm - lane: the warp's first row)
      uint16_t* at = reinterpret_cast<uint16_t*>(yrow + gn0) + (int64_t)((lane >> 4) - lane) * p.ldy + col;
#pragma unroll 4
      for (int i = 0; i < 16; ++i, at += 2 * p.ldy) {
        const int r = 2 * i + (lane >> 4);
        const uint16_t x = stage[r * 16 + ((col >> 3) ^ ((r >> 2) & 1)) * 8 + (col & 7)];
        if (r < rows && col < valid) *at = x;
      }
      __syncwarp();
    } else if (gm < p.M) {
      store_row16<TOut>(yrow + gn0, v, valid, vec);
    }
  }
}

// B_MN is a template parameter because the K-major kernel must not pay for the other layout: with a run-time test of it in the
// MMA and load loops 8 products of [65536, 256] x [256, 128] took 78 us, 74 without.
// Y: how results leave, one kernel each: with two of them in one, whole tiles took 3 % longer ([65536, 88] x [88, 176] fp16 12.7 us,
// 13.0), with three 14 %, by spills. map_y is read where that is by TMA.
enum { Y_PIECES, Y_TMA, Y_ANY };
template <typename TOut, bool B_MN, int Y>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_umma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_y, const __grid_constant__ UmmaGemmParams p) {
  using namespace umma;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int b_stage_bytes = (B_MN ? (p.block_n + 63) / 64 * 64 : p.block_n) * BLOCK_K * 2;
  uint8_t* smem_a = smem;
  const int STAGES = p.stages;
  uint8_t* smem_b = smem + STAGES * A_STAGE_BYTES;      // per-stage B tiles, or the resident B tile (all k blocks)
  __shared__ __align__(8) uint64_t b_full, b_free;
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
  // tile numbers fit 31 bits (checked by the host): 32-bit divisions, a few per tile and thread
  const uint32_t tiles_mn = (uint32_t)p.tiles_m * (uint32_t)p.tiles_n;
  const uint32_t total_tiles = tiles_mn * (uint32_t)p.batch;
  const uint32_t acc_stride = (uint32_t)p.tmem_cols / 2;
  // A tile's place: m fastest, or (n_fast, rings only) n fastest, so that the n tiles of one row of tiles run at the same
  // time and its A rows come from HBM once.
  auto place = [&](uint32_t tile, int& b, int& m0, int& n0) {
    b = (int)(tile / tiles_mn);
    const uint32_t rem = tile - (uint32_t)b * tiles_mn, inner = (uint32_t)(p.n_fast ? p.tiles_n : p.tiles_m), o = rem / inner, i = rem - o * inner;
    m0 = (int)(p.n_fast ? o : i) * BLOCK_M;
    n0 = (int)(p.n_fast ? i : o) * p.block_n;
  };
  // Tile sequence of this CTA, the same for every role. With a resident B tile each CTA takes a contiguous
  // run (m fastest), so that B changes once or twice per CTA; otherwise CTAs interleave, so that the CTAs
  // running at the same time read the same B tile from L2.
  const bool bres = p.b_resident != 0;
  const uint32_t tile_first = bres ? blockIdx.x * p.tiles_per_cta : blockIdx.x;
  const uint32_t tile_step = bres ? 1u : gridDim.x;
  const uint32_t tile_end = bres ? min(total_tiles, tile_first + p.tiles_per_cta) : total_tiles;
  const int b_bytes_per_load = bres ? 0 : b_stage_bytes;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&b_full), 1);
    mbar_init(smem_u32(&b_free), 1);
    for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&full_bar[s]), 1); mbar_init(smem_u32(&empty_bar[s]), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&acc_full[s]), 1); mbar_init(smem_u32(&acc_empty[s]), EPI_WARPS); }
    fence_barrier_init();
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
    if (Y == Y_TMA) prefetch_tensormap(&map_y);
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_base_s), (uint32_t)p.tmem_cols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      // one k block of B: one box of block_n rows x 64 k, or (N-major) boxes of 64 k rows x 64 columns side by side
      auto load_b = [&](uint32_t dst, uint32_t bar, int kb, int n0, int b) {
        if (!B_MN) {
          tma_load_3d(dst, &map_b, bar, kb * BLOCK_K, n0, b);
        } else {
          for (int j = 0; j * 64 < p.block_n; ++j) tma_load_3d(dst + j * MN_BOX_BYTES, &map_b, bar, n0 + j * 64, kb * BLOCK_K, b);
        }
      };
      int s = 0;
      uint32_t ph = 0;                 // stage and its phase: the stage counter wraps, the phase flips
      uint32_t b_loads = 0;
      int cur_n0 = -1, cur_b = -1;
      bool ok = true;
      for (uint32_t tile = tile_first; tile < tile_end && ok; tile += tile_step) {
        int b, m0, n0;
        place(tile, b, m0, n0);
        if (bres && (n0 != cur_n0 || b != cur_b)) {
          cur_n0 = n0; cur_b = b;
          // the MMAs that read the previous B tile have completed (signalled after the last tile that used it)
          if (b_loads > 0) ok = mbar_wait(smem_u32(&b_free), (b_loads - 1) & 1u, 5);
          if (!ok) break;
          mbar_arrive_expect_tx(smem_u32(&b_full), (uint32_t)(num_kb * b_stage_bytes));
          for (int kb = 0; kb < num_kb; ++kb)
            load_b(smem_u32(smem_b + kb * b_stage_bytes), smem_u32(&b_full), kb, n0, p.b_batched ? b : 0);
          ++b_loads;
        }
        for (int kb = 0; kb < num_kb; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
          ok = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, 1);
          if (!ok) break;
          mbar_arrive_expect_tx(smem_u32(&full_bar[s]), (uint32_t)(A_STAGE_BYTES + b_bytes_per_load));
          tma_load_3d(smem_u32(smem_a + s * A_STAGE_BYTES), &map_a, smem_u32(&full_bar[s]), kb * BLOCK_K, m0,
                      p.a_batched ? b : 0);
          if (!bres) load_b(smem_u32(smem_b + s * b_stage_bytes), smem_u32(&full_bar[s]), kb, n0, p.b_batched ? b : 0);
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp runs the issue loop in uniform control flow and one elected lane issues: the descriptors then
    // live in uniform registers, which is what the MMA instruction reads, and the issue cost per MMA drops to about
    // a third of what one thread under `if (lane == 0)` pays.
    {
      int s = 0, it = 0;
      uint32_t ph = 0;
      uint32_t b_loads = 0;
      uint32_t cur_bn = 0xffffffffu;             // (batch, n tile) of the resident B tile
      bool ok = true;
      for (uint32_t tile = tile_first; tile < tile_end && ok; tile += tile_step, ++it) {
        const int as = it & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_empty[as]), ((uint32_t)(it >> 1) & 1u) ^ 1u, 4));   // epilogue drained it
        if (!ok) break;
        if (bres && tile / (uint32_t)p.tiles_m != cur_bn) {
          cur_bn = tile / (uint32_t)p.tiles_m;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&b_full), b_loads & 1u, 6));
          if (!ok) break;
          ++b_loads;
        }
        tc_fence_after_sync();
        const uint32_t tmem_acc = tmem_base + as * acc_stride;
        for (int kb = 0; kb < num_kb; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[s]), ph, 2));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(smem_a + s * A_STAGE_BYTES);
          const uint32_t b_addr = smem_u32(smem_b + (bres ? kb : s) * b_stage_bytes);
#pragma unroll
          for (int k = 0; k < BLOCK_K / 16; ++k) {
            const uint64_t da = make_desc_sw128(a_addr + k * 32, 1024);
            const uint64_t db = B_MN ? make_desc_sw128_mn(b_addr + k * 2048, MN_BOX_BYTES) : make_desc_sw128(b_addr + k * 32, 1024);
            mma_f16_ss_elect(tmem_acc, da, db, p.idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          mma_commit_elect(smem_u32(&empty_bar[s]));     // slot free once these MMAs have read it
        }
        mma_commit_elect(smem_u32(&acc_full[as]));       // accumulator complete
        // the next tile of this CTA needs another B tile: tell the producer when these MMAs are done with this one
        if (bres && ok && tile + tile_step < tile_end && (tile + tile_step) / (uint32_t)p.tiles_m != cur_bn)
          mma_commit_elect(smem_u32(&b_free));
      }
    }
  } else {
    // epilogue: warp w may touch TMEM lanes [32*(w%4), 32*(w%4)+32); the four warpgroups split the columns.
    // Per-column operands (bias, activation parameters) are staged in shared memory once per (n tile,
    // batch) - a persistent CTA walks m tiles first, so that is rare - and each thread loads all the
    // accumulator chunks it owns before it waits, so one TMEM round trip is exposed per tile.
    const int ew = warp - 2;
    const int q = warp & 3;
    const int part = ew >> 2;
    const int row = q * 32 + lane;
    const int chunks = p.block_n / 16;
    const int c_begin = chunks * part / 4, c_end = chunks * (part + 1) / 4;
    const bool vec_base = ((reinterpret_cast<uintptr_t>(p.Y) & 15) == 0) && ((p.ldy * sizeof(TOut)) % 16 == 0) &&
                          ((p.stride_y * sizeof(TOut)) % 16 == 0);
    float* s_bias = reinterpret_cast<float*>(smem + STAGES * A_STAGE_BYTES +
                                             (bres ? num_kb : STAGES) * b_stage_bytes);           // [4][256]
    uint4* stage = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s_bias + 4 * 256) + ew * EPI_STAGE_BYTES);
    float* s_a = s_bias + 256;
    float* s_b = s_a + 256;
    float* s_c = s_b + 256;
    int it = 0, cur_n0 = -1, cur_b = -1;
    bool ok = true;
    uint8_t* area = Y == Y_TMA ? reinterpret_cast<uint8_t*>(s_bias + 4 * 256) + ew * p.y_bufs * p.y_unit * 64 : nullptr;
    uint32_t turn = 0;                                        // units that this warp has stored
    // A warp whose accumulator wait ran out keeps walking the tile sequence without touching tensor memory,
    // global memory or the acc_empty barrier: the other epilogue warps may have passed the same wait (each
    // lane keeps its own clock), and they still need this warp at the two named barriers below.
    for (uint32_t tile = tile_first; tile < tile_end; tile += tile_step, ++it) {
      int b, m0, n0;
      place(tile, b, m0, n0);
      const int as = it & 1;
      const int gm = m0 + row;
      if (n0 != cur_n0 || b != cur_b) {
        cur_n0 = n0; cur_b = b;
        asm volatile("bar.sync 2, 512;" ::: "memory");                  // everyone is done with the old columns
        const int e = ew * 32 + lane, gn = n0 + e;
        if (e < p.block_n) stage_columns(p, b, gn, e, s_bias, s_a, s_b, s_c);
        asm volatile("bar.sync 2, 512;" ::: "memory");
      }
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[as]), (uint32_t)(it >> 1) & 1u, 3));
      if (!ok) continue;
      tc_fence_after_sync();
      const uint32_t tmem_acc = tmem_base + as * acc_stride + ((uint32_t)(q * 32) << 16);
      if constexpr (Y == Y_TMA) {
        const int y = m0 + q * 32, cols = min(p.block_n, p.N - n0), y1 = p.y_beside ? b : y, y2 = p.y_beside ? y : b;
        with_kind(p.epi.kind, [&](auto kind) {
          constexpr int KIND = decltype(kind)::value;
          if (p.y_unit == 32)
            epi_tile_tma<TOut, KIND, 32>(map_y, tmem_acc, part, cols, p.alpha, s_bias, s_a, s_b, s_c, area, p.y_bufs, turn, n0, y1, y2, y < p.M, lane);
          else
            epi_tile_tma<TOut, KIND, 16>(map_y, tmem_acc, part, cols, p.alpha, s_bias, s_a, s_b, s_c, area, p.y_bufs, turn, n0, y1, y2, y < p.M, lane);
        });
      } else {
        TOut* yrow = reinterpret_cast<TOut*>(p.Y) + (int64_t)b * p.stride_y + (int64_t)gm * p.ldy;
        // fp32: whole tiles without a check at each piece, the others element by element ([65536, 64] x [64, 64] 11.3 us, 9.4;
        // 8 x ([4096, 256] x [256, 128]) 13.2, 11.1; [65536, 200] x [200, 80] 17.4, 14.5)
        if (sizeof(TOut) == 4 && Y == Y_PIECES && m0 + BLOCK_M <= p.M && n0 + p.block_n <= p.N) {
          with_kind(p.epi.kind, [&](auto kind) {
            epi_tile_fast<TOut, decltype(kind)::value, true>(tmem_acc, c_begin, c_end, p.alpha, s_bias, s_a, s_b, s_c, yrow + n0, p.ldy, 32, p.block_n, stage, lane);
          });
        } else if constexpr (Y == Y_ANY || sizeof(TOut) == 4) {
          const int brow = p.bias_group > 1 ? (int)((uint32_t)gm / (uint32_t)p.bias_group) : gm;   // bias row of this output row
          epi_tile_edge<TOut>(p, tmem_acc, c_begin, c_end, s_bias, s_a, s_b, s_c, yrow, b, gm, brow, n0, vec_base,
                              reinterpret_cast<uint16_t*>(stage), lane);
        } else {
          const int rows = p.M - (m0 + q * 32), cols = p.N - n0;
          with_kind(p.epi.kind, [&](auto kind) {
            epi_tile_fast<TOut, decltype(kind)::value>(tmem_acc, c_begin, c_end, p.alpha, s_bias, s_a, s_b, s_c, yrow + n0, p.ldy, rows, cols, stage, lane);
          });
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty[as]));              // one arrival per epilogue warp
    }
    if (Y == Y_TMA && lane == 0) tma_store_wait_read<0>();
  }

  pdl_release();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// [batch, rows, K] tensor of 2-byte elements, box {box_cols, box_rows, box_batch}, swizzled over the box's row (an N-major B is the same with
// its k rows as rows and its columns as the inner extent; so is Y)
int make_map(CUtensorMap* map, const void* base, int is_bf16, int64_t K, int64_t rows, int64_t ld, int64_t batch,
             int64_t batch_stride, int box_rows, int box_cols = BLOCK_K, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, int box_batch = 1) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(XB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)(batch > 1 ? batch_stride : ld * rows) * 2};
  if (strides[1] == 0) strides[1] = strides[0];
  cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, (cuuint32_t)box_batch};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(XB_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  return 0;
}

// Columns of a tile: all of a product of up to 256, equal shares of a wider one (128 columns each until it
// was so: [65536, 24] x [24, 272] fp16, three tiles of which the last held 16 columns, 18.9 us, 15.5 as two of 144); narrower (down to 32, or to the 64 of a box of an
// N-major B) where the tiles would leave SMs idle: a CTA's time is the latency of its operand stream, which shrinks with the
// tile, and A comes from L2 for every column of tiles. 8 products of
// [1000, 256] x [256, 128] fp16 (64 tiles of 128 columns, 128 of 64): 6.8 -> 5.8 us.
int pick_block_n(const xb_gemm_args& a) {
  const int wide = (a.N + 255) / 256, bn = ((a.N + wide - 1) / wide + 15) / 16 * 16;
  const int64_t rows = ((int64_t)a.M + BLOCK_M - 1) / BLOCK_M * a.batch;
  const int least = a.trans_b ? 32 : 64;
  const int64_t split = std::min<int64_t>(sm_count() / std::max<int64_t>(rows, 1), (a.N + least - 1) / least);
  if (split <= (a.N + bn - 1) / bn) return bn;
  return (int)((a.N + split - 1) / split + 15) / 16 * 16;
}

bool umma_eligible(const xb_gemm_args& a) {
  if (a.ab_dtype != XB_F16 && a.ab_dtype != XB_BF16) return false;
  if (a.trans_a) return false;
  if (a.y_dtype != XB_F16 && a.y_dtype != XB_BF16 && a.y_dtype != XB_F32) return false;
  // [K, N] weights with fp32 results stay on the CUDA cores: the tensor cores do not round every partial sum, which a 16-bit
  // result hides (the same error against 64 bits from both engines, 2.07e-4 fp16 and 1.66e-3 bf16) and an fp32 one does not
  // (K = 512: 6.4e-7 against 3.9e-7 with fp16 operands, 4.7e-7 against 1.6e-7 with bf16 ones).
  if (!a.trans_b && a.y_dtype == XB_F32) return false;
  if (a.lda % 8 || a.ldb % 8 || a.stride_a % 8 || a.stride_b % 8) return false;
  if ((reinterpret_cast<uintptr_t>(a.A) & 15) || (reinterpret_cast<uintptr_t>(a.B) & 15)) return false;
  if (a.lda < a.K || a.ldb < (a.trans_b ? a.K : a.N)) return false;
  return true;
}

template <typename TOut, bool B_MN, int Y>
int launch_umma(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& my, const UmmaGemmParams& p, dim3 grid, size_t smem,
                cudaStream_t s) {
  static PerDeviceOnce attr_set;   // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr_set, SMEM_BUDGET + 6 * 1024, (const void*)gemm_umma_kernel<TOut, B_MN, Y>);
  launch_dependent(gemm_umma_kernel<TOut, B_MN, Y>, grid, GEMM_THREADS, smem, s, ma, mb, my, p);
  return check_launch("gemm_umma_kernel");
}
template <typename TOut, bool B_MN>
int launch_umma_half(int y, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& my, const UmmaGemmParams& p, dim3 grid, size_t smem,
                     cudaStream_t s) {
  if (y == Y_TMA) return launch_umma<TOut, B_MN, Y_TMA>(ma, mb, my, p, grid, smem, s);
  if (y == Y_PIECES) return launch_umma<TOut, B_MN, Y_PIECES>(ma, mb, mb, p, grid, smem, s);
  return launch_umma<TOut, B_MN, Y_ANY>(ma, mb, mb, p, grid, smem, s);
}

void fill_umma_params(UmmaGemmParams& p, const xb_gemm_args& a) {
  memset(&p, 0, sizeof(p));
  p.M = a.M; p.N = a.N; p.K = a.K;
  p.block_n = pick_block_n(a);
  p.tmem_cols = 64;                                      // two accumulator stages, each at least 32 columns
  while (p.tmem_cols < 2 * p.block_n) p.tmem_cols <<= 1;
  p.alpha = a.alpha; p.beta = a.beta;
  p.a_batched = a.stride_a != 0; p.b_batched = a.stride_b != 0;
  p.bias = a.bias; p.ldbias = a.ldbias; p.stride_bias = a.stride_bias;
  p.bias_group = a.bias_row_group > 1 ? (int)a.bias_row_group : 1;
  p.bias_kind = a.bias ? a.bias_kind : XB_BIAS_NONE; p.bias_dtype = a.bias_dtype;
  p.Y = a.Y; p.ldy = a.ldy; p.stride_y = a.stride_y; p.y_dtype = a.y_dtype;
  p.epi.kind = a.epilogue; p.epi.a = a.ep_a; p.epi.b = a.ep_b; p.epi.c = a.ep_c;
  p.epi.count = a.ep_count; p.epi.nosqrt = a.dice_nosqrt; p.stride_ep = a.stride_ep;
  p.batch = a.batch;
  p.b_mn = !a.trans_b;
  p.idesc = umma::make_idesc(BLOCK_M, p.block_n, a.ab_dtype == XB_BF16) | (p.b_mn ? umma::IDESC_B_MN : 0u);
}

// Where the batches of Y lie: one after the other, or beside one another in its rows (an axis-1 concat).
bool y_stacked(const xb_gemm_args& a) { return a.batch == 1 || a.stride_y >= (int64_t)a.M * a.ldy; }
bool y_beside(const xb_gemm_args& a) { return !y_stacked(a) && a.stride_y >= a.N && a.stride_y * a.batch <= a.ldy; }
// map of a two-byte Y for copies of 32 rows x `unit` columns
int make_y_map(CUtensorMap* map, const xb_gemm_args& a, int unit) {
  const CUtensorMapSwizzle sw = unit == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
  const int bf = a.y_dtype == XB_BF16;
  return y_beside(a) ? make_map(map, a.Y, bf, a.N, a.batch, a.stride_y, a.M, a.ldy, 1, unit, sw, 32)
                     : make_map(map, a.Y, bf, a.N, a.M, a.ldy, a.batch, a.stride_y, 32, unit, sw);
}

// Two-CTA tiles where they fill the chip (a 256 x 256 tile for every pair of SMs) and the epilogue is the plain one: whole
// 256-column tiles, aligned output rows, no bias matrix. Below that the one-CTA kernel spreads the work over more SMs.
// [65536, 1280] x [1280, 1024] and the two layers after it (bf16): 207 us as pairs, 290 one CTA at a time. Less depth than 384 is
// an epilogue with a few MMAs beside it, and the one-CTA kernel has two staging areas a warp (65536 rows, N = 512: K = 256 26.8 us,
// 31.3 as pairs; 320 29.9, 33.7; 384 33.4, 35.1; 448 37.3, 36.3; 640 48.9, 44.0. 20000 rows: 13.5, 13.9; 14.9, 14.8; 16.3, 15.4).
bool pair_wanted(const xb_gemm_args& a) {
  const int64_t es = a.y_dtype == XB_F32 ? 4 : 2;
  return a.trans_b && a.N % 256 == 0 && a.K >= (es == 4 ? 256 : 384) && !(a.bias && a.bias_kind == XB_BIAS_FULL) &&
         (reinterpret_cast<uintptr_t>(a.Y) & 15) == 0 && (a.ldy * es) % 16 == 0 && (a.stride_y * es) % 16 == 0 &&
         ((int64_t)a.M + 255) / 256 * (a.N / 256) * a.batch >= sm_count() / 2 && (es == 4 || y_stacked(a) || y_beside(a));
}

}  // namespace
}  // namespace xb

#include "xb_gemm_umma_pair.cuh"

namespace xb {
namespace {

template <typename TOut>
int launch_umma_pair(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& my, const UmmaGemmParams& p, dim3 grid, size_t smem,
                     cudaStream_t s) {
  static PerDeviceOnce attr_set;   // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr_set, 226 * 1024, (const void*)gemm_umma_pair_kernel<TOut>);
  launch_dependent(gemm_umma_pair_kernel<TOut>, grid, GEMM_THREADS, smem, s, ma, mb, my, p);
  return check_launch("gemm_umma_pair_kernel");
}

int gemm_umma(const xb_gemm_args& a, cudaStream_t stream) {
  UmmaGemmParams p;
  fill_umma_params(p, a);
  const int is_bf16 = a.ab_dtype == XB_BF16;
  CUtensorMap ma, mb, my;
  if (int rc = make_map(&ma, a.A, is_bf16, a.K, a.M, a.lda, p.a_batched ? a.batch : 1, a.stride_a, BLOCK_M)) return rc;
  // after the ring: per-column epilogue parameters [4][256] fp32, then the epilogue warps' staging areas
  int tail = 4 * 256 * (int)sizeof(float) + (a.y_dtype == XB_F32 ? 0 : EPI_WARPS * EPI_STAGE_BYTES);
  if (pair_wanted(a) && (a.y_dtype == XB_F32 || make_y_map(&my, a, 32) == 0)) {
    p.y_unit = 32; p.y_bufs = PAIR_Y_BUFS; p.y_beside = y_beside(a);
    tail = 4 * 256 * (int)sizeof(float) + (a.y_dtype == XB_F32 ? 0 : EPI_WARPS * PAIR_Y_BUFS * 32 * 64);
    if (int rc = make_map(&mb, a.B, is_bf16, a.K, a.N, a.ldb, p.b_batched ? a.batch : 1, a.stride_b, PAIR_N / 2)) return rc;
    p.tiles_m = (a.M + 2 * BLOCK_M - 1) / (2 * BLOCK_M);
    p.tiles_n = a.N / PAIR_N;
    p.idesc = umma::make_idesc(2 * BLOCK_M, PAIR_N, is_bf16);
    p.stages = std::min(PAIR_MAX_STAGES, (225 * 1024 - tail) / PAIR_STAGE_BYTES);
    const size_t smem = (size_t)p.stages * PAIR_STAGE_BYTES + tail + 1024;
    const int64_t total = (int64_t)p.tiles_m * p.tiles_n * p.batch;
    XB_REQUIRE(total < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gemm: %lld output tiles are too many for one call", (long long)total);
    const dim3 grid(2 * (unsigned)std::min<int64_t>(total, sm_count() / 2));
    switch (a.y_dtype) {
      case XB_F16: return launch_umma_pair<__half>(ma, mb, my, p, grid, smem, stream);
      case XB_BF16: return launch_umma_pair<__nv_bfloat16>(ma, mb, my, p, grid, smem, stream);
      default: return launch_umma_pair<float>(ma, mb, mb, p, grid, smem, stream);
    }
  }
  if (int rc = p.b_mn ? make_map(&mb, a.B, is_bf16, a.N, a.K, a.ldb, p.b_batched ? a.batch : 1, a.stride_b, BLOCK_K)
                      : make_map(&mb, a.B, is_bf16, a.K, a.N, a.ldb, p.b_batched ? a.batch : 1, a.stride_b, p.block_n))
    return rc;
  p.tiles_m = (a.M + BLOCK_M - 1) / BLOCK_M;
  p.tiles_n = (a.N + p.block_n - 1) / p.block_n;
  const int64_t total = (int64_t)p.tiles_m * p.tiles_n * p.batch;
  XB_REQUIRE(total < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gemm: %lld output tiles are too many for one call", (long long)total);
  // Rows of whole, aligned 16-byte pieces, and no bias matrix; those by TMA where a CTA has several tiles. (One tile is a chain of
  // latencies that the copy lengthens: 2 x ([1862, 88] x [88, 24]) bf16 3.5 us, 3.9 by TMA; [1000, 88] x [88, 168] fp16 3.8 and 4.0.)
  const int64_t es = a.y_dtype == XB_F32 ? 4 : 2;
  const bool pieces = p.bias_kind != XB_BIAS_FULL && (reinterpret_cast<uintptr_t>(a.Y) & 15) == 0 && a.ldy * es % 16 == 0 &&
                      (a.batch == 1 || a.stride_y * es % 16 == 0) && a.N * es % 16 == 0;
  int y = pieces ? Y_PIECES : Y_ANY;
  if (pieces && es == 2 && total > sm_count() && (y_stacked(a) || y_beside(a))) {
    // copies of 32 columns, 16 where the tile has few or where 32 would reach into the next tile
    p.y_unit = p.block_n >= 128 && (p.block_n % 32 == 0 || p.tiles_n == 1) ? 32 : 16;
    p.y_bufs = p.block_n > 4 * p.y_unit ? 2 : 1;
    p.y_beside = y_beside(a);
    if (make_y_map(&my, a, p.y_unit) == 0) {
      y = Y_TMA;
      tail = 4 * 256 * (int)sizeof(float) + EPI_WARPS * p.y_bufs * p.y_unit * 64;
    }
  }
  // persistent: one CTA per SM walks the tiles; the accumulator is double-buffered in TMEM so the
  // epilogue of one tile overlaps the loads and MMAs of the next
  dim3 grid((unsigned)std::min<int64_t>(total, sm_count()));
  // When the whole B tile (all of K) is small and several m tiles share it, it is loaded once and stays in
  // shared memory: re-reading it from L2 for every tile doubles the L2-to-SM traffic of a thin GEMM, which
  // then bounds the kernel below the HBM rate.
  const int b_stage_bytes = (p.b_mn ? (p.block_n + 63) / 64 * 64 : p.block_n) * BLOCK_K * 2;
  const int num_kb = (a.K + BLOCK_K - 1) / BLOCK_K;
  const int grid_ctas = (int)std::min<int64_t>(total, sm_count());
  p.tiles_per_cta = (uint32_t)((total + grid_ctas - 1) / grid_ctas);
  p.b_resident = (int64_t)num_kb * b_stage_bytes <= 96 * 1024 && p.tiles_m >= 4 && p.tiles_per_cta >= 2;
  // n first where the CTAs that run together then share A rows instead of fetching them again for every n tile (the whole
  // weight matrix stays in L2 either way at the sizes of a dense tower); m first where A fits L2 itself, since a CTA then
  // keeps its columns and stages their parameters once. (A of the 65536-row tower's first
  // layer is 168 MB and was read four times.)
  p.n_fast = !p.b_resident && p.tiles_n > 1 && (int64_t)a.M * a.K * 2 > (32 << 20) && (int64_t)a.N * a.K * 2 <= (32 << 20);
  const int k_blocks = (int)std::min<int64_t>((int64_t)num_kb * p.tiles_per_cta, MAX_STAGES);      // of one CTA's whole walk
  size_t smem;
  if (p.b_resident) {
    const int b_bytes = num_kb * b_stage_bytes;
    p.stages = std::max(2, std::min({MAX_STAGES, (SMEM_BUDGET - tail - b_bytes) / A_STAGE_BYTES, k_blocks}));
    smem = (size_t)p.stages * A_STAGE_BYTES + b_bytes + tail + 1024;
  } else {
    const int stage_bytes = A_STAGE_BYTES + b_stage_bytes;
    p.stages = std::max(2, std::min({MAX_STAGES, (SMEM_BUDGET - tail) / stage_bytes, k_blocks}));
    smem = (size_t)p.stages * stage_bytes + tail + 1024;
  }
  switch (a.y_dtype) {
    case XB_F16:
      return p.b_mn ? launch_umma_half<__half, true>(y, ma, mb, my, p, grid, smem, stream) : launch_umma_half<__half, false>(y, ma, mb, my, p, grid, smem, stream);
    case XB_BF16:
      return p.b_mn ? launch_umma_half<__nv_bfloat16, true>(y, ma, mb, my, p, grid, smem, stream)
                    : launch_umma_half<__nv_bfloat16, false>(y, ma, mb, my, p, grid, smem, stream);
    default:                                             // (never b_mn: umma_eligible)
      return y == Y_PIECES ? launch_umma<float, false, Y_PIECES>(ma, mb, mb, p, grid, smem, stream)
                           : launch_umma<float, false, Y_ANY>(ma, mb, mb, p, grid, smem, stream);
  }
}

}  // namespace

int gemm_umma_status(int* out) { return umma::read_status_word(out); }
int gemm_umma_clear_status() { return umma::clear_status_word(); }

}  // namespace xb

using namespace xb;

namespace xb {
int att_status(int* out);
int att_clear_status();
int tower_status(int* out);
int tower_clear_status();
int att_set_status_mirror(int* p);
int tower_set_status_mirror(int* p);
int rnn_status(int* out);
int rnn_clear_status();
int rnn_set_status_mirror(int* p);

// Host-mapped copy of the status word, one per device: {host address, device address}.
struct StatusMirror { volatile int* host = nullptr; int* dev = nullptr; };
static StatusMirror g_mirror[64];
static std::mutex g_mirror_mu;
}  // namespace xb

// A wait that nothing will ever satisfy, with its own short limit: shows that a bounded wait gives up,
// records where, and leaves the context usable. Site code 99.
__global__ void wait_selftest_kernel(long long limit_cycles) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    umma::mbar_init(umma::smem_u32(&bar), 1);
    umma::fence_barrier_init();
  }
  __syncthreads();
  const long long t0 = clock64();
  bool done = false;
  while (!(done = umma::mbar_try_wait(umma::smem_u32(&bar), 0))) {
    if (clock64() - t0 > limit_cycles) break;
  }
  if (!done && threadIdx.x == 0) umma::wait_gave_up(99);
}

extern "C" int xb_selftest_wait_timeout(int64_t limit_cycles, xb_stream_t stream) {
  XB_REQUIRE(limit_cycles > 0 && limit_cycles <= ((int64_t)1 << 31), XB_ERR_ARG,
             "xb_selftest_wait_timeout: limit of %lld cycles (1 .. 2^31)", (long long)limit_cycles);
  wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((long long)limit_cycles);
  return check_launch("wait_selftest_kernel");
}

extern "C" int xb_device_status(int* status) {
  XB_REQUIRE(status, XB_ERR_ARG, "xb_device_status: null pointer");
  int a = 0, b = 0, c = 0, d = 0;
  XB_REQUIRE(gemm_umma_status(&a) == 0 && att_status(&b) == 0 && tower_status(&c) == 0 && rnn_status(&d) == 0, XB_ERR_CUDA,
             "xb_device_status: read failed");
  *status = a ? a : (b ? b : (c ? c : d));
  return 0;
}

extern "C" int xb_device_status_clear(void) {
  XB_REQUIRE(gemm_umma_clear_status() == 0 && att_clear_status() == 0 && tower_clear_status() == 0 && rnn_clear_status() == 0, XB_ERR_CUDA,
             "xb_device_status_clear failed");
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lock(g_mirror_mu);
    if (g_mirror[dev].host) *g_mirror[dev].host = 0;
  }
  return 0;
}

extern "C" int xb_device_status_mirror(const volatile int** host_word) {
  XB_REQUIRE(host_word, XB_ERR_ARG, "xb_device_status_mirror: null pointer");
  int dev = 0;
  XB_CUDA(cudaGetDevice(&dev));
  XB_REQUIRE(dev >= 0 && dev < 64, XB_ERR_LIMIT, "xb_device_status_mirror: device ordinal %d", dev);
  std::lock_guard<std::mutex> lock(g_mirror_mu);
  StatusMirror& m = g_mirror[dev];
  if (m.host == nullptr) {
    int* h = nullptr;
    int* d = nullptr;
    XB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&h), 64, cudaHostAllocMapped | cudaHostAllocPortable));
    *h = 0;
    if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&d), h, 0) != cudaSuccess) {
      cudaFreeHost(h);
      return fail(XB_ERR_CUDA, "xb_device_status_mirror: cudaHostGetDevicePointer failed");
    }
    if (umma::set_status_mirror(d) != 0 || att_set_status_mirror(d) != 0 || tower_set_status_mirror(d) != 0 ||
        rnn_set_status_mirror(d) != 0) {
      umma::set_status_mirror(nullptr); att_set_status_mirror(nullptr); tower_set_status_mirror(nullptr);
      rnn_set_status_mirror(nullptr);
      cudaFreeHost(h);
      return fail(XB_ERR_CUDA, "xb_device_status_mirror: could not publish the mirror address");
    }
    // a wait may have run out before the mirror existed
    int now = 0;
    if (xb_device_status(&now) == 0) *h = now;
    m.host = h;
    m.dev = d;
  }
  *host_word = m.host;
  return 0;
}

static int validate_gemm(const xb_gemm_args* a) {
  XB_REQUIRE(a, XB_ERR_ARG, "xb_gemm: null arguments");
  XB_REQUIRE(a->M >= 0 && a->N >= 0 && a->K >= 0 && a->batch >= 0, XB_ERR_ARG, "xb_gemm: negative size");
  XB_REQUIRE(a->A && a->B && a->Y, XB_ERR_ARG, "xb_gemm: null matrix");
  XB_REQUIRE(a->ab_dtype == XB_F32 || a->ab_dtype == XB_F16 || a->ab_dtype == XB_BF16, XB_ERR_UNSUPPORTED,
             "xb_gemm: operand dtype %d", a->ab_dtype);
  XB_REQUIRE(a->y_dtype == XB_F32 || a->y_dtype == XB_F16 || a->y_dtype == XB_BF16, XB_ERR_UNSUPPORTED,
             "xb_gemm: output dtype %d", a->y_dtype);
  XB_REQUIRE(a->epilogue >= XB_EPI_NONE && a->epilogue <= XB_EPI_SIGMOID, XB_ERR_UNSUPPORTED,
             "xb_gemm: epilogue %d", a->epilogue);
  XB_REQUIRE(a->epilogue != XB_EPI_PRELU || (a->ep_a && (a->ep_count == 1 || a->ep_count == a->N)), XB_ERR_ARG,
             "xb_gemm: PRelu needs 1 or N slopes");
  XB_REQUIRE(a->epilogue != XB_EPI_DICE || (a->ep_a && a->ep_b && a->ep_c), XB_ERR_ARG,
             "xb_gemm: Dice needs gamma, mean and var");
  XB_REQUIRE(!a->bias || a->bias_kind == XB_BIAS_ROW || a->bias_kind == XB_BIAS_FULL, XB_ERR_ARG,
             "xb_gemm: bias kind %d", a->bias_kind);
  XB_REQUIRE(!a->bias || dtype_size(a->bias_dtype) != 0, XB_ERR_UNSUPPORTED, "xb_gemm: bias dtype %d", a->bias_dtype);
  XB_REQUIRE(a->bias_row_group >= 0 && (a->bias_row_group <= 1 || (a->bias && a->bias_kind == XB_BIAS_FULL)), XB_ERR_ARG,
             "xb_gemm: bias_row_group needs a full [rows, N] bias");
  const int64_t a_cols = a->trans_a ? a->M : a->K, b_cols = a->trans_b ? a->K : a->N;
  XB_REQUIRE(a->lda >= a_cols && a->ldb >= b_cols && a->ldy >= a->N, XB_ERR_ARG,
             "xb_gemm: leading dimension smaller than the row (lda=%lld ldb=%lld ldy=%lld)", (long long)a->lda,
             (long long)a->ldb, (long long)a->ldy);
  return 0;
}

// Whether XB_GEMM_AUTO runs these arguments on the tcgen05 engine.
// Less than 128 x 64 outputs keep sums that are rounded, fp32 FMAs or gemm_half_kernel's, whose error against 64 bits is no larger;
// an accumulator in tensor memory is cut off at every MMA instead (rms before the result's rounding, positive fp16 values 5.6e-7,
// FMAs 1.3e-7). What that costs: 16 x ([22, 320] x [320, 16]) fp16 8.0 us, 4.3 in tensor memory (30 on the CUDA cores);
// 2 x ([59, 24] x [24, 32]) 3.6, 3.2 (5.5); K-major [1, 1280] x [1280, 512] 21, 7.9 (90).
static bool auto_takes_umma(const xb_gemm_args& a) {
  return umma_eligible(a) && a.K > 0 && !gemm_narrow_takes(a) && (int64_t)a.M * a.N * a.batch >= 128 * 64;
}

extern "C" int xb_gemm_uses_tcgen05(const xb_gemm_args* a) {
  if (!a || (a->engine != XB_GEMM_AUTO && a->engine != XB_GEMM_TCGEN05)) return 0;
  if (a->engine == XB_GEMM_TCGEN05) return a->trans_b && a->K > 0 && umma_eligible(*a) ? 1 : 0;
  return auto_takes_umma(*a) ? 1 : 0;
}

extern "C" int xb_gemm(const xb_gemm_args* a, xb_stream_t stream) {
  if (int rc = validate_gemm(a)) return rc;
  if (a->M == 0 || a->N == 0 || a->batch == 0) return 0;
  if (a->engine == XB_GEMM_TCGEN05) {
    XB_REQUIRE(a->trans_b && umma_eligible(*a), XB_ERR_UNSUPPORTED,
               "xb_gemm: tcgen05 engine needs fp16/bf16, A [M,K] and B [N,K] row-major, 16-byte aligned, "
               "leading dimensions and batch strides multiples of 8");
    XB_REQUIRE(a->K > 0, XB_ERR_ARG, "xb_gemm: K = 0");
    return gemm_umma(*a, (cudaStream_t)stream);
  }
  if (a->engine == XB_GEMM_AUTO && auto_takes_umma(*a)) return gemm_umma(*a, (cudaStream_t)stream);
  return gemm_simt(*a, (cudaStream_t)stream);
}
