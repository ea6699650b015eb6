// CUDA-core GEMM engine with the fused bias/activation epilogue.
//
// Serves what the tcgen05 engine does not take: fp32 operands (the reference's
// 1e-6 operator fixtures need true fp32 products, not tf32), transposed A,
// leading dimensions that break TMA's 16-byte rule, and tiny shapes.
//
// 256 threads as 16 x 16, TM x TN outputs each (tile 16*TM x 16*TN), 16-deep k
// slices double-buffered in shared memory, the next slice on its way to
// registers while the current one is multiplied; fp32 accumulation with k
// ascending, whatever the tile.
// What bounds it is the FMA rate where the launch fills the chip: a thread reads
// TM values of A as 16-byte vectors (two addresses a warp: a broadcast) and TN
// scalars of B for TM*TN FMAs, so the shared-memory pipe stays below the FMA
// pipe from 8 x 4 up. [50000, 144] x [144, 80] fp32
// with Dice: 114 us, 230 with the 64 x 64 tile of 4 x 4 outputs this replaces (a second column of tiles three
// quarters empty, four scalar reads of each operand for 16 FMAs).
#include "xb_common.cuh"

namespace xb {

struct SimtGemmParams {
  int tiles_n;
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

template <int TM, int TN>
__global__ void __launch_bounds__(256, TM * TN >= 40 ? 2 : 3) gemm_simt_kernel(const __grid_constant__ SimtGemmParams p) {
  pdl_begin();
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

  EpiParams epi = p.epi;
  if (epi.a) epi.a += (int64_t)b * p.stride_ep;
  if (epi.b) epi.b += (int64_t)b * p.stride_ep;
  if (epi.c) epi.c += (int64_t)b * p.stride_ep;
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int gn = n0 + tx + 16 * j;
    if (gn >= p.N) continue;
    const float rb = p.bias_kind == XB_BIAS_ROW ? load_as_f32(p.bias, (int64_t)b * p.stride_bias + gn, p.bias_dtype) : 0.f;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + ty * TM + i;
      if (gm >= p.M) continue;
      float v = p.alpha * acc[i][j];
      if (p.bias_kind == XB_BIAS_ROW)
        v += p.beta * rb;
      else if (p.bias_kind == XB_BIAS_FULL)
        v += p.beta * load_as_f32(p.bias, (int64_t)b * p.stride_bias + (int64_t)(gm / p.bias_group) * p.ldbias + gn, p.bias_dtype);
      v = apply_epilogue(epi, v, gn);
      store_from_f32(p.Y, (int64_t)b * p.stride_y + (int64_t)gm * p.ldy + gn, p.y_dtype, v);
    }
  }
}

template <int TM>
static void launch_simt_tm(const SimtGemmParams& p, int tn, dim3 grid, cudaStream_t s) {
  switch (tn) {
    case 1: launch_dependent(gemm_simt_kernel<TM, 1>, grid, 256, 0, s, p); break;
    case 2: launch_dependent(gemm_simt_kernel<TM, 2>, grid, 256, 0, s, p); break;
    case 3: launch_dependent(gemm_simt_kernel<TM, 3>, grid, 256, 0, s, p); break;
    case 4: launch_dependent(gemm_simt_kernel<TM, 4>, grid, 256, 0, s, p); break;
    case 5: launch_dependent(gemm_simt_kernel<TM, 5>, grid, 256, 0, s, p); break;
    case 6: launch_dependent(gemm_simt_kernel<TM, 6>, grid, 256, 0, s, p); break;
    default: launch_dependent(gemm_simt_kernel<TM, 8>, grid, 256, 0, s, p); break;
  }
}

// Tile of a product: a wave of CTAs costs what its busiest SM computes, TM*TN a k slice and output pair, plus what
// the operand reads and the slice's overhead cost beside it; the tile with the cheapest sum of waves is taken.
static void pick_simt_tile(int64_t M, int64_t N, int64_t batch, int* tm, int* tn) {
  double best = 0;
  for (int m : {8, 4, 2}) {
    for (int n : {8, 6, 5, 4, 3, 2, 1}) {
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
  int tm = 8, tn = 8;
  pick_simt_tile(a.M, a.N, a.batch, &tm, &tn);
  XB_REQUIRE((a.M + 63) / 64 <= 65535 && a.batch <= 65535, XB_ERR_LIMIT, "xb_gemm: M or batch too large for the SIMT engine");
  p.tiles_n = (a.N + 16 * tn - 1) / (16 * tn);
  const int64_t tiles = (((int64_t)a.M + 16 * tm - 1) / (16 * tm)) * p.tiles_n;
  XB_REQUIRE(tiles < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gemm: %lld output tiles are too many for one call", (long long)tiles);
  dim3 grid((unsigned)tiles, (unsigned)a.batch);
  if (tm == 8) launch_simt_tm<8>(p, tn, grid, stream);
  else if (tm == 4) launch_simt_tm<4>(p, tn, grid, stream);
  else launch_simt_tm<2>(p, tn, grid, stream);
  return check_launch("gemm_simt_kernel");
}

}  // namespace xb
