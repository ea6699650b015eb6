// CUDA-core GEMM engine with the fused bias/activation epilogue.
//
// Serves what the tcgen05 engine does not take: fp32 operands (the reference's
// 1e-6 operator fixtures need true fp32 products, not tf32) and fp32 results of
// 16-bit operands in the layouts and sizes that it leaves. (16-bit results of
// those go through warp-level matrix instructions, xb_gemm_half.cuh.)
//
// 256 threads, tile 16*TM x 16*TN, 16-deep k slices; fp32 accumulation with k
// ascending, whatever the tile, so every form gives the same bits. XB_GEMM_SIMT
// is these tiles; XB_GEMM_AUTO also takes the kernels for a few columns and for
// batches of single rows, which add up partial sums.
// gemm_f32_kernel (fp32, neither operand transposed: Blaze's own layout) keeps
// a ring of slices in flight with cp.async, which hides the latency that bounds
// a small launch, and puts two columns' FMAs into one fma.rn.f32x2 (each
// rounded as an FMA of its own), so that a thread owns pairs of adjacent
// columns. Its outputs leave through shared memory in a rolled loop: what
// bounded it was the fetching of code that was unrolled over them.
// [50000, 144] x [144, 80]: 42 us (75 with unrolled outputs, 114 with the
// general kernel's register prefetch); [8192, 512] x [512, 512]: 117 us,
// 37 TFLOP/s (150); 45 TFLOP/s of 72 at K = 4096.
// gemm_simt_kernel is the general form: any type, layout and alignment, the next
// slice on its way to registers while the current one is multiplied.
#include <algorithm>

#include "xb_common.cuh"

namespace xb {

struct SimtGemmParams {
  int tiles_n, y_pairs;
  int M, N, K, trans_a, trans_b, in_dtype, y_dtype, a_vec, b_vec;
  float alpha, beta;
  const void* A; int64_t lda, stride_a;
  const void* B; int64_t ldb, stride_b;
  const void* bias; int64_t ldbias, stride_bias, bias_group; int bias_kind, bias_dtype;
  void* Y; int64_t ldy, stride_y;
  EpiParams epi; int64_t stride_ep;
};

constexpr int SIMT_BK = 16;

// One operand's slice of `ROWS` rows (m or n) x 16 k on its way from global to shared memory. `kmaj`: k is the
// contiguous direction (a row's k elements are adjacent), otherwise the rows are. Element e of a thread's share is
// (row, k) by the maps below, so that neighbouring threads read neighbouring addresses in either direction.
template <int ROWS>
struct SimtSlice {
  static constexpr int PER = (ROWS * SIMT_BK + 255) / 256;      // elements per thread
  static constexpr int VPER = (ROWS * SIMT_BK / 4 + 255) / 256; // 16-byte pieces per thread
  static constexpr int PITCH = ROWS + 4;                        // shared memory row of one k: 16-byte aligned
  float v[VPER * 4 > PER ? VPER * 4 : PER];

  __device__ __forceinline__ void load(const void* base, int64_t ld, int row0, int rows, int k0, int K, bool kmaj, bool vec, int dt) {
    if (vec) {                                                  // fp32, 16-byte aligned, extent a multiple of 4
      const float* f = reinterpret_cast<const float*>(base);
#pragma unroll
      for (int i = 0; i < VPER; ++i) {
        const int q = threadIdx.x + i * 256;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ROWS * SIMT_BK / 4 % 256 == 0 || q < ROWS * SIMT_BK / 4) {
          const int r = kmaj ? q / (SIMT_BK / 4) : q % (ROWS / 4) * 4, k = kmaj ? q % (SIMT_BK / 4) * 4 : q / (ROWS / 4);
          if (row0 + r < rows && k0 + k < K)
            x = __ldg(reinterpret_cast<const float4*>(kmaj ? f + (int64_t)(row0 + r) * ld + k0 + k : f + (int64_t)(k0 + k) * ld + row0 + r));
        }
        v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int q = threadIdx.x + i * 256;
        v[i] = 0.f;
        if (ROWS * SIMT_BK % 256 == 0 || q < ROWS * SIMT_BK) {
          const int r = kmaj ? q / SIMT_BK : q % ROWS, k = kmaj ? q % SIMT_BK : q / ROWS;
          if (row0 + r < rows && k0 + k < K)
            v[i] = load_as_f32(base, kmaj ? (int64_t)(row0 + r) * ld + k0 + k : (int64_t)(k0 + k) * ld + row0 + r, dt);
        }
      }
    }
  }
  __device__ __forceinline__ void store(float* s, bool kmaj, bool vec) const {
    if (vec) {
#pragma unroll
      for (int i = 0; i < VPER; ++i) {
        const int q = threadIdx.x + i * 256;
        if (ROWS * SIMT_BK / 4 % 256 == 0 || q < ROWS * SIMT_BK / 4) {
          const int r = kmaj ? q / (SIMT_BK / 4) : q % (ROWS / 4) * 4, k = kmaj ? q % (SIMT_BK / 4) * 4 : q / (ROWS / 4);
          if (kmaj) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[(k + e) * PITCH + r] = v[4 * i + e];
          } else {
            *reinterpret_cast<float4*>(s + k * PITCH + r) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int q = threadIdx.x + i * 256;
        if (ROWS * SIMT_BK % 256 == 0 || q < ROWS * SIMT_BK)
          s[(kmaj ? q % SIMT_BK : q / ROWS) * PITCH + (kmaj ? q / SIMT_BK : q % ROWS)] = v[i];
      }
    }
  }
};

// What an output column needs beside its sum, read once per thread and column; then bias and activation of one output.
struct Column { float bias, a, b, c; };
__device__ __forceinline__ Column column_of(const SimtGemmParams& p, int b, int gn) {
  Column o = {0.f, 0.f, 0.f, 0.f};
  const int64_t eo = (int64_t)b * p.stride_ep + gn;
  if (p.bias_kind == XB_BIAS_ROW) o.bias = load_as_f32(p.bias, (int64_t)b * p.stride_bias + gn, p.bias_dtype);
  if (p.epi.kind == XB_EPI_PRELU) o.a = p.epi.a[p.epi.count == 1 ? (int64_t)b * p.stride_ep : eo];
  if (p.epi.kind == XB_EPI_DICE) { o.a = p.epi.a[eo]; o.b = p.epi.b[eo]; o.c = dice_rstd(p.epi.c[eo], p.epi.nosqrt); }
  return o;
}
__device__ __forceinline__ float finish(const SimtGemmParams& p, const Column& c, int b, int gm, int gn, float acc) {
  float v = p.alpha * acc;
  if (p.bias_kind == XB_BIAS_ROW)
    v += p.beta * c.bias;
  else if (p.bias_kind == XB_BIAS_FULL)
    v += p.beta * load_as_f32(p.bias, (int64_t)b * p.stride_bias + (int64_t)(gm / p.bias_group) * p.ldbias + gn, p.bias_dtype);
  if (p.epi.kind == XB_EPI_PRELU) return act_prelu(v, c.a);
  if (p.epi.kind == XB_EPI_DICE) return act_dice(v, c.a, c.b, c.c);
  if (p.epi.kind == XB_EPI_SIGMOID) return act_sigmoid(v);
  return v;
}

// (one copy of the code: see the outputs of gemm_f32_kernel)
__device__ __noinline__ void finish_and_store(const SimtGemmParams& p, Column c, int b, int gm, int gn, float acc) {
  store_from_f32(p.Y, (int64_t)b * p.stride_y + (int64_t)gm * p.ldy + gn, p.y_dtype, finish(p, c, b, gm, gn, acc));
}

template <int TM, int TN>
__global__ void __launch_bounds__(256, TM * TN >= 40 ? 2 : 3) gemm_simt_kernel(const __grid_constant__ SimtGemmParams p) {
  pdl_wait();
  constexpr int BM = 16 * TM, BN = 16 * TN;
  using SliceA = SimtSlice<BM>;
  using SliceB = SimtSlice<BN>;
  __shared__ __align__(16) float As[2][SIMT_BK * SliceA::PITCH];
  __shared__ __align__(16) float Bs[2][SIMT_BK * SliceB::PITCH];
  const int b = blockIdx.y;
  const size_t es = p.in_dtype == XB_F32 ? 4 : 2;
  const char* A = reinterpret_cast<const char*>(p.A) + (int64_t)b * p.stride_a * es;
  const char* B = reinterpret_cast<const char*>(p.B) + (int64_t)b * p.stride_b * es;
  // neighbouring CTAs take the n tiles of one m tile: its rows come from L2 after the first
  const int mt = blockIdx.x / p.tiles_n, m0 = mt * BM, n0 = (int)(blockIdx.x - (unsigned)mt * p.tiles_n) * BN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const bool a_kmaj = !p.trans_a, b_kmaj = p.trans_b != 0, a_vec = p.a_vec != 0, b_vec = p.b_vec != 0;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  SliceA sa;
  SliceB sb;
  const int nk = (p.K + SIMT_BK - 1) / SIMT_BK;
  if (nk > 0) {
    sa.load(A, p.lda, m0, p.M, 0, p.K, a_kmaj, a_vec, p.in_dtype);
    sb.load(B, p.ldb, n0, p.N, 0, p.K, b_kmaj, b_vec, p.in_dtype);
    sa.store(As[0], a_kmaj, a_vec);
    sb.store(Bs[0], b_kmaj, b_vec);
  }
  __syncthreads();
  for (int kb = 0; kb < nk; ++kb) {
    const bool more = kb + 1 < nk;
    if (more) {
      sa.load(A, p.lda, m0, p.M, (kb + 1) * SIMT_BK, p.K, a_kmaj, a_vec, p.in_dtype);
      sb.load(B, p.ldb, n0, p.N, (kb + 1) * SIMT_BK, p.K, b_kmaj, b_vec, p.in_dtype);
    }
    const float* as = As[kb & 1] + ty * TM;
    const float* bs = Bs[kb & 1] + tx;
#pragma unroll
    for (int k = 0; k < SIMT_BK; ++k) {
      float a[TM], bb[TN];
      if constexpr (TM >= 4) {
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
          const float4 x = *reinterpret_cast<const float4*>(as + k * SliceA::PITCH + i);
          a[i] = x.x; a[i + 1] = x.y; a[i + 2] = x.z; a[i + 3] = x.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = as[k * SliceA::PITCH + i];
      }
#pragma unroll
      for (int j = 0; j < TN; ++j) bb[j] = bs[k * SliceB::PITCH + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], bb[j], acc[i][j]);
    }
    if (more) {
      sa.store(As[(kb + 1) & 1], a_kmaj, a_vec);     // last read before the barrier of the previous slice
      sb.store(Bs[(kb + 1) & 1], b_kmaj, b_vec);
      __syncthreads();
    }
  }

  pdl_release();
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int gn = n0 + tx + 16 * j;
    if (gn >= p.N) continue;
    const Column c = column_of(p, b, gn);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + ty * TM + i;
      if (gm < p.M) finish_and_store(p, c, b, gm, gn, acc[i][j]);
    }
  }
}

// fp32, A [M, K] and B [K, N] as they lie. A ring of F32_STAGES slices: A as [row][k] (pitch 20: a warp's two rows on other
// banks), B as [k][column]; 16-byte copies where the operand's rows allow, 4-byte ones otherwise, zeros past the edges.
constexpr int F32_STAGES = 4, F32_APITCH = SIMT_BK + 4;
template <int TM, int TN>
struct F32Tile {
  static constexpr int BM = 16 * TM, BN = 16 * TN, A_FLOATS = BM * F32_APITCH, B_FLOATS = SIMT_BK * BN;
  static constexpr int SMEM = F32_STAGES * (A_FLOATS + B_FLOATS) * 4;
  static_assert(BM * BN * 4 <= SMEM, "the ring also holds the tile's outputs");
};
__device__ __forceinline__ void cp_async_zfill16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_zfill4(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}

template <int TM, int TN>
__global__ void __launch_bounds__(256, TM * TN >= 40 ? 2 : 3) gemm_f32_kernel(const __grid_constant__ SimtGemmParams p) {
  using Tl = F32Tile<TM, TN>;
  extern __shared__ __align__(16) float ring[];
  pdl_wait();
  const int b = blockIdx.y;
  const float* A = reinterpret_cast<const float*>(p.A) + (int64_t)b * p.stride_a;
  const float* B = reinterpret_cast<const float*>(p.B) + (int64_t)b * p.stride_b;
  const int mt = blockIdx.x / p.tiles_n, m0 = mt * Tl::BM, n0 = (int)(blockIdx.x - (unsigned)mt * p.tiles_n) * Tl::BN;
  const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;          // rows ty + 32 i, columns 2 tx + 16 j and the next
  const int nk = (p.K + SIMT_BK - 1) / SIMT_BK;
  const uint32_t ring_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(ring));

  auto request = [&](int kb) {
    if (kb < nk) {
      const int k0 = kb * SIMT_BK;
      const uint32_t as = ring_u32 + (kb % F32_STAGES) * (Tl::A_FLOATS + Tl::B_FLOATS) * 4, bs = as + Tl::A_FLOATS * 4;
      if (p.a_vec) {
#pragma unroll
        for (int q0 = 0; q0 < Tl::BM * 4; q0 += 256) {
          const int q = q0 + threadIdx.x;
          if (Tl::BM * 4 % 256 == 0 || q < Tl::BM * 4) {
            const int r = q / 4, k = q % 4 * 4;
            const bool in = m0 + r < p.M && k0 + k < p.K;
            cp_async_zfill16(as + (r * F32_APITCH + k) * 4, in ? A + (int64_t)(m0 + r) * p.lda + k0 + k : A, in);
          }
        }
      } else {
        for (int q = threadIdx.x; q < Tl::BM * SIMT_BK; q += 256) {
          const int r = q / SIMT_BK, k = q % SIMT_BK;
          const bool in = m0 + r < p.M && k0 + k < p.K;
          cp_async_zfill4(as + (r * F32_APITCH + k) * 4, in ? A + (int64_t)(m0 + r) * p.lda + k0 + k : A, in);
        }
      }
      if (p.b_vec) {
#pragma unroll
        for (int q0 = 0; q0 < Tl::BN * 4; q0 += 256) {
          const int q = q0 + threadIdx.x;
          if (Tl::BN * 4 % 256 == 0 || q < Tl::BN * 4) {
            const int k = q / (Tl::BN / 4), n = q % (Tl::BN / 4) * 4;
            const bool in = n0 + n < p.N && k0 + k < p.K;
            cp_async_zfill16(bs + (k * Tl::BN + n) * 4, in ? B + (int64_t)(k0 + k) * p.ldb + n0 + n : B, in);
          }
        }
      } else {
        for (int q = threadIdx.x; q < Tl::BN * SIMT_BK; q += 256) {
          const int k = q / Tl::BN, n = q % Tl::BN;
          const bool in = n0 + n < p.N && k0 + k < p.K;
          cp_async_zfill4(bs + (k * Tl::BN + n) * 4, in ? B + (int64_t)(k0 + k) * p.ldb + n0 + n : B, in);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");        // an empty group keeps the count
  };

  constexpr int R = TM / 2;                                     // rows of a thread
  uint64_t acc[R][TN];                                          // pairs of fp32
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  // one copy of `request`: this loop asks for the first slices too
#pragma unroll 1
  for (int kb = 1 - F32_STAGES; kb < nk; ++kb) {
    if (kb < 0) {
      request(kb + F32_STAGES - 1);
      continue;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
    __syncthreads();                                            // slice kb has landed; slice kb - 1 has been read
    request(kb + F32_STAGES - 1);
    const float* as = ring + (kb % F32_STAGES) * (Tl::A_FLOATS + Tl::B_FLOATS) + ty * F32_APITCH;
    const float* bs = ring + (kb % F32_STAGES) * (Tl::A_FLOATS + Tl::B_FLOATS) + Tl::A_FLOATS + 2 * tx;
#pragma unroll
    for (int k4 = 0; k4 < SIMT_BK; k4 += 4) {
      float a[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(as + 32 * i * F32_APITCH + k4);
        a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint64_t bb[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) bb[j] = *reinterpret_cast<const uint64_t*>(bs + (k4 + k) * Tl::BN + 16 * j);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          uint64_t aa;
          asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i][k]));
#pragma unroll
          for (int j = 0; j < TN; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(bb[j]));
        }
      }
    }
  }
  // Outputs go through shared memory (the ring is done with), so that bias, activation and store are one rolled loop: unrolled
  // over a thread's outputs they are some 100 KB of code that every SM fetches to run once, 40 us whatever K.
  pdl_release();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) *reinterpret_cast<uint64_t*>(ring + (ty + 32 * i) * Tl::BN + 2 * tx + 16 * j) = acc[i][j];
  __syncthreads();
  constexpr int PAIRS = Tl::BN / 2, STEP = 256 / PAIRS;         // a thread keeps its two columns and takes every STEP-th row
  const int cp = threadIdx.x % PAIRS, r0 = threadIdx.x / PAIRS, gn = n0 + 2 * cp;
  if (r0 >= STEP || gn >= p.N) return;
  const bool two = gn + 1 < p.N;
  const Column c0 = column_of(p, b, gn), c1 = column_of(p, b, two ? gn + 1 : gn);
#pragma unroll 1
  for (int r = r0; r < Tl::BM && m0 + r < p.M; r += STEP) {
    const int gm = m0 + r;
    const float2 x = *reinterpret_cast<const float2*>(ring + r * Tl::BN + 2 * cp);
    const float v0 = finish(p, c0, b, gm, gn, x.x), v1 = two ? finish(p, c1, b, gm, gn + 1, x.y) : 0.f;
    const int64_t at = (int64_t)b * p.stride_y + (int64_t)gm * p.ldy + gn;
    if (p.y_pairs && two) {
      *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.Y) + at) = make_float2(v0, v1);
    } else {
      store_from_f32(p.Y, at, p.y_dtype, v0);
      if (two) store_from_f32(p.Y, at + 1, p.y_dtype, v1);
    }
  }
}

template <int TM, int TN>
static int launch_f32(const SimtGemmParams& p, dim3 grid, cudaStream_t s) {
  static PerDeviceOnce attr;                                    // per instantiation
  if (F32Tile<TM, TN>::SMEM > 48 * 1024) XB_SET_MAX_SMEM_ONCE(attr, (F32Tile<TM, TN>::SMEM), (const void*)gemm_f32_kernel<TM, TN>);
  launch_dependent(gemm_f32_kernel<TM, TN>, grid, 256, F32Tile<TM, TN>::SMEM, s, p);
  return check_launch("gemm_f32_kernel");
}
template <int TM>
static int launch_f32_tm(const SimtGemmParams& p, int tn, dim3 grid, cudaStream_t s) {
  switch (tn) {
    case 1: return launch_f32<TM, 1>(p, grid, s);
    case 2: return launch_f32<TM, 2>(p, grid, s);
    case 3: return launch_f32<TM, 3>(p, grid, s);
    case 4: return launch_f32<TM, 4>(p, grid, s);
    case 5: return launch_f32<TM, 5>(p, grid, s);
    case 6: return launch_f32<TM, 6>(p, grid, s);
    default: return launch_f32<TM, 8>(p, grid, s);
  }
}
template <int TM>
static int launch_simt_tm(const SimtGemmParams& p, int tn, dim3 grid, cudaStream_t s) {
  switch (tn) {
    case 2: launch_dependent(gemm_simt_kernel<TM, 2>, grid, 256, 0, s, p); break;
    case 4: launch_dependent(gemm_simt_kernel<TM, 4>, grid, 256, 0, s, p); break;
    default: launch_dependent(gemm_simt_kernel<TM, 8>, grid, 256, 0, s, p); break;
  }
  return check_launch("gemm_simt_kernel");
}

}  // namespace xb
#include "xb_gemm_half.cuh"
namespace xb {

// ---- batches of single rows (fp32): the weighted sum of an attention unit run operator by operator -------------------------
// A tile has 32 rows at the least and a batch of such products one row each: here a CTA takes a batch, its threads four
// columns of every few k, and the partial sums are added in order. Bound by the read of B. 500 x ([1, 100] x [100, 36]):
// 4.5 us, 20 in tiles.
__global__ void __launch_bounds__(256) gemm_f32_row_kernel(const __grid_constant__ SimtGemmParams p) {
  extern __shared__ __align__(16) float part[];                 // [groups][N]
  pdl_wait();
  const int b = blockIdx.x, N4 = p.N / 4, groups = 256 / N4, g = threadIdx.x / N4, c = threadIdx.x - g * N4;
  const float* A = reinterpret_cast<const float*>(p.A) + (int64_t)b * p.stride_a;
  const float* B = reinterpret_cast<const float*>(p.B) + (int64_t)b * p.stride_b;
  if (g < groups) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = g; k0 < p.K; k0 += 4 * groups) {
      float a[4];
      float4 w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u * groups;
        const bool in = k < p.K;
        a[u] = in ? __ldg(A + k) : 0.f;
        w[u] = in ? __ldg(reinterpret_cast<const float4*>(B + (int64_t)k * p.ldb) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc.x = fmaf(a[u], w[u].x, acc.x); acc.y = fmaf(a[u], w[u].y, acc.y);
        acc.z = fmaf(a[u], w[u].z, acc.z); acc.w = fmaf(a[u], w[u].w, acc.w);
      }
    }
    *reinterpret_cast<float4*>(part + g * p.N + 4 * c) = acc;
  }
  __syncthreads();
  pdl_release();
  for (int n = threadIdx.x; n < p.N; n += 256) {
    float v = part[n];
    for (int i = 1; i < groups; ++i) v += part[i * p.N + n];
    store_from_f32(p.Y, (int64_t)b * p.stride_y + n, p.y_dtype, finish(p, column_of(p, b, n), b, 0, n, v));
  }
}

// ---- one to four output columns: the last layer of a tower or of an attention unit, a stream over A ----------------------
// A tile of either GEMM engine computes 16 columns at the least and reads A through a ring made for tiles that are used many
// times. Here `lanes` lanes share a row, each with every lanes-th 16-byte piece of it (up to four, requested together, those
// of the next row before this one's are used), the weights lie in shared memory as fp32, and the lanes' sums meet by shuffles.
//
// Bound by the read of A. [1000, 512] x [512, 4] fp16: 39 us on the tensor cores (one tile walks all of K eight times over), 11 here with
// the call; [50000, 40] x [40, 1] fp32: 7.4 us after the kernel before, 5.3; [65536, 256] x [256, 1] the same either way.
constexpr int NARROW_N = 4, NARROW_PIECES = 4;
template <typename T, int N>
__global__ void __launch_bounds__(256) gemm_narrow_kernel(const __grid_constant__ SimtGemmParams p, int lanes) {
  constexpr int E = 16 / (int)sizeof(T);                        // elements of a piece
  extern __shared__ __align__(16) float ws[];                   // [N][K]
  __shared__ Column cols[N];
  pdl_wait();
  const int b = blockIdx.y, K = p.K, pieces = K / E;
  const T* A = reinterpret_cast<const T*>(p.A) + (int64_t)b * p.stride_a;
  const T* B = reinterpret_cast<const T*>(p.B) + (int64_t)b * p.stride_b;
  const int l = threadIdx.x & (lanes - 1), team = threadIdx.x / lanes, teams = 256 / lanes;
  const int64_t step = (int64_t)gridDim.x * teams;
  auto request = [&](int64_t r, uint4 (&raw)[NARROW_PIECES]) {
    const uint4* row = reinterpret_cast<const uint4*>(A + r * p.lda);
#pragma unroll
    for (int i = 0; i < NARROW_PIECES; ++i) {
      const int c = l + i * lanes;
      raw[i] = r < p.M && c < pieces ? __ldg(row + c) : make_uint4(0, 0, 0, 0);
    }
  };
  uint4 raw[NARROW_PIECES], next[NARROW_PIECES];                // (the first rows are on their way before the weights)
  request((int64_t)blockIdx.x * teams + team, raw);
  for (int i = threadIdx.x; i < N * K; i += 256) {
    const int n = i / K, k = i - n * K;
    ws[i] = n < p.N ? to_f32<T>(p.trans_b ? B[(int64_t)n * p.ldb + k] : B[(int64_t)k * p.ldb + n]) : 0.f;
  }
  if ((int)threadIdx.x < p.N) cols[threadIdx.x] = column_of(p, b, threadIdx.x);
  __syncthreads();
  pdl_release();
  // (every lane of a warp walks as many rows, so that the shuffles are whole)
  for (int64_t r0 = (int64_t)blockIdx.x * teams; r0 < p.M; r0 += step) {
    const int64_t r = r0 + team;
    request(r + step, next);
    float acc[N];
#pragma unroll
    for (int n = 0; n < N; ++n) acc[n] = 0.f;
#pragma unroll
    for (int i = 0; i < NARROW_PIECES; ++i) {
      const int c = l + i * lanes;
      if (c >= pieces) break;
      const T* a = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
      for (int n = 0; n < N; ++n) {
#pragma unroll
        for (int e = 0; e < E; e += 4) {
          const float4 w = *reinterpret_cast<const float4*>(ws + n * K + c * E + e);
          acc[n] = fmaf(to_f32<T>(a[e]), w.x, acc[n]);
          acc[n] = fmaf(to_f32<T>(a[e + 1]), w.y, acc[n]);
          acc[n] = fmaf(to_f32<T>(a[e + 2]), w.z, acc[n]);
          acc[n] = fmaf(to_f32<T>(a[e + 3]), w.w, acc[n]);
        }
      }
    }
    for (int off = lanes >> 1; off > 0; off >>= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) acc[n] += __shfl_xor_sync(0xffffffffu, acc[n], off);
    }
#pragma unroll
    for (int i = 0; i < NARROW_PIECES; ++i) raw[i] = next[i];
    if (r >= p.M) continue;
#pragma unroll
    for (int n = 0; n < N; ++n)
      if (n < p.N && n % lanes == l)
        store_from_f32(p.Y, (int64_t)b * p.stride_y + r * p.ldy + n, p.y_dtype, finish(p, cols[n], b, (int)r, n, acc[n]));
  }
}

// What gemm_narrow_kernel takes: whole 16-byte pieces, aligned, and as many rows as the tiles take. (Fewer rows than fill a few
// blocks gain nothing.)
bool gemm_narrow_takes(const xb_gemm_args& a) {
  const int E = a.ab_dtype == XB_F32 ? 4 : 8;
  return a.N <= NARROW_N && !a.trans_a && a.M >= 128 && a.M <= 65535 * 64 && a.K > 0 && a.K % E == 0 && a.K / E <= 32 * NARROW_PIECES &&
         a.lda % E == 0 && a.stride_a % E == 0 && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0 && a.batch <= 65535;
}

template <typename T>
static int launch_narrow(const SimtGemmParams& p, int batch, cudaStream_t s) {
  const int pieces = p.K * (int)sizeof(T) / 16;
  int lanes = 1;
  while (lanes * NARROW_PIECES < pieces) lanes <<= 1;
  const int64_t blocks = std::min<int64_t>(((int64_t)p.M * lanes + 255) / 256, (int64_t)sm_count() * 4);
  const dim3 grid((unsigned)blocks, (unsigned)batch);
  const int n = p.N == 3 ? 4 : p.N;
  const size_t smem = (size_t)n * p.K * 4;
  if (n == 1) launch_dependent(gemm_narrow_kernel<T, 1>, grid, 256, smem, s, p, lanes);
  else if (n == 2) launch_dependent(gemm_narrow_kernel<T, 2>, grid, 256, smem, s, p, lanes);
  else launch_dependent(gemm_narrow_kernel<T, 4>, grid, 256, smem, s, p, lanes);
  return check_launch("gemm_narrow_kernel");
}

// Tile of a product: a wave of CTAs costs what its busiest SM computes, TM*TN a k slice and output pair, plus what
// the operand reads (1.5 TN + 0.75 TM) and the slice's barrier and index work (4) cost beside it; the tile with the cheapest sum
// of waves is taken. The three weights are estimates in units of FMAs, not fitted to measurements of each tile. The general
// kernel has fewer widths.
static void pick_simt_tile(int64_t M, int64_t N, int64_t batch, bool f32, int* tm, int* tn) {
  double best = 0;
  for (int m : {8, 4, 2}) {
    for (int n : {8, 6, 5, 4, 3, 2, 1}) {
      if (!f32 && n != 8 && n != 4 && n != 2) continue;
      const int64_t tiles = ((M + 16 * m - 1) / (16 * m)) * ((N + 16 * n - 1) / (16 * n)) * batch;
      const double waves = (double)((tiles + sm_count() - 1) / sm_count());
      const double cost = waves * (m * n + 1.5 * n + 0.75 * m + 4);
      if (best == 0 || cost < best) { best = cost; *tm = m; *tn = n; }
    }
  }
}

int gemm_simt(const xb_gemm_args& a, cudaStream_t stream) {
  SimtGemmParams p;
  p.M = a.M; p.N = a.N; p.K = a.K; p.trans_a = a.trans_a; p.trans_b = a.trans_b;
  p.in_dtype = a.ab_dtype; p.y_dtype = a.y_dtype;
  p.alpha = a.alpha; p.beta = a.beta;
  p.A = a.A; p.lda = a.lda; p.stride_a = a.stride_a;
  p.B = a.B; p.ldb = a.ldb; p.stride_b = a.stride_b;
  p.bias = a.bias; p.ldbias = a.ldbias; p.stride_bias = a.stride_bias;
  p.bias_group = a.bias_row_group > 1 ? a.bias_row_group : 1;
  p.bias_kind = a.bias ? a.bias_kind : XB_BIAS_NONE; p.bias_dtype = a.bias_dtype;
  p.Y = a.Y; p.ldy = a.ldy; p.stride_y = a.stride_y;
  p.epi.kind = a.epilogue; p.epi.a = a.ep_a; p.epi.b = a.ep_b; p.epi.c = a.ep_c;
  p.epi.count = a.ep_count; p.epi.nosqrt = a.dice_nosqrt; p.stride_ep = a.stride_ep;
  // 16-byte loads of fp32 operands: every vector aligned and, along the contiguous direction, wholly inside
  auto vec = [&](const void* ptr, int64_t ld, int64_t stride, int64_t extent) {
    return a.ab_dtype == XB_F32 && (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && ld % 4 == 0 && stride % 4 == 0 && extent % 4 == 0;
  };
  p.a_vec = vec(a.A, a.lda, a.stride_a, a.trans_a ? a.M : a.K);
  p.b_vec = vec(a.B, a.ldb, a.stride_b, a.trans_b ? a.K : a.N);
  p.y_pairs = a.y_dtype == XB_F32 && (reinterpret_cast<uintptr_t>(a.Y) & 7) == 0 && a.ldy % 2 == 0 && a.stride_y % 2 == 0;
  int tm = 8, tn = 8;
  const bool f32 = a.ab_dtype == XB_F32 && !a.trans_a && !a.trans_b;
  pick_simt_tile(a.M, a.N, a.batch, f32, &tm, &tn);
  // (the entry point's limits, whatever the tile; a grid of any of them would take more rows)
  XB_REQUIRE((a.M + 63) / 64 <= 65535 && a.batch <= 65535, XB_ERR_LIMIT, "xb_gemm: M or batch too large for the SIMT engine");
  // Who asks for this engine by name gets its order of sums; the kernels from here to the tiles have others.
  const bool any = a.engine == XB_GEMM_AUTO;
  // single rows: many of them, each of a size that one CTA reads in a few steps
  if (any && f32 && a.M == 1 && a.batch >= 32 && a.N % 4 == 0 && a.N <= 256 && (int64_t)a.N * a.K <= 65536 && p.b_vec) {
    launch_dependent(gemm_f32_row_kernel, (unsigned)a.batch, 256, (size_t)(256 / (a.N / 4)) * a.N * 4, stream, p);
    return check_launch("gemm_f32_row_kernel");
  }
  if (any && gemm_narrow_takes(a)) {
    if (a.ab_dtype == XB_F32) return launch_narrow<float>(p, a.batch, stream);
    if (a.ab_dtype == XB_F16) return launch_narrow<__half>(p, a.batch, stream);
    return launch_narrow<__nv_bfloat16>(p, a.batch, stream);
  }
  // 16-bit results of 16-bit operands: sums of 16 products by matrix instructions, which are no further from 64 bits than FMAs.
  // (Their bits differ from the FMAs', which an fp32 result would show.) One slice of up to 16 k is quicker on the CUDA cores unless
  // there are more columns than a tile and many outputs: K = 14, us there and here: [706, 14] x [14, 43] 4.5, 6.0,
  // [46002, 14] x [14, 15] 9.6, 11.6, [42, 14] x [14, 119] 4.6, 5.8, [1087, 3] x [3, 121] 4.8, 6.3; 4 x ([3001, 14] x [14, 65]) 12.6, 9.1, [20000, 14] x [14, 255] 36, 25;
  // K = 17: 5.4, 6.2; 12.9, 11.9; 5.6, 6.1; 16, 9.6; 46, 26.
  const bool shallow = a.K <= 16 && (a.N <= 64 || (int64_t)a.M * a.N * a.batch < 1 << 18);
  if (any && a.ab_dtype != XB_F32 && a.y_dtype != XB_F32 && !shallow) return gemm_half(p, a, stream);
  p.tiles_n = (a.N + 16 * tn - 1) / (16 * tn);
  const int64_t tiles = (((int64_t)a.M + 16 * tm - 1) / (16 * tm)) * p.tiles_n;
  XB_REQUIRE(tiles < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gemm: %lld output tiles are too many for one call", (long long)tiles);
  dim3 grid((unsigned)tiles, (unsigned)a.batch);
  if (f32) return tm == 8 ? launch_f32_tm<8>(p, tn, grid, stream) : tm == 4 ? launch_f32_tm<4>(p, tn, grid, stream) : launch_f32_tm<2>(p, tn, grid, stream);
  return tm == 8 ? launch_simt_tm<8>(p, tn, grid, stream) : tm == 4 ? launch_simt_tm<4>(p, tn, grid, stream) : launch_simt_tm<2>(p, tn, grid, stream);
}

}  // namespace xb
