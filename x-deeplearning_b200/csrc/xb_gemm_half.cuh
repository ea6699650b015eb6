// 16-bit products that the tcgen05 engine does not take: rows that TMA cannot address (odd leading dimensions, operands that
// start anywhere), transposed A and less than 128 x 64 outputs. Included by xb_gemm_simt.cu.
//
// Warp-level matrix instructions on operands that the threads fetch themselves: a warp reads 64 adjacent elements of a row, a lane
// two of them, with one 4-byte load where the rows allow it and two 2-byte loads otherwise, the next slice of 64 k in registers
// while this one is multiplied. fp32 accumulation; the outputs leave through shared memory, whole rows of 64.
//
// Bound by the issue of these narrow loads where the product is large, by the latency of the slices where it is small (up to K / 64
// trips to memory one after the other). fp16, on the CUDA cores before and here: [30000, 500] x [500, 511] 1125 -> 146 us (rows of
// A at 4-byte addresses, N = 512: 1131 -> 120), [30000, 313] x [313, 31] 90 -> 16, 8 x ([2254, 117] x [117, 144]) 69 -> 19,
// 2 x ([47350, 28] x [28, 27]) bf16 with a sigmoid 30 -> 22 (12 us more where narrow rows do not share a warp),
// 2 x ([2585, 67] x [67, 45]) 23 -> 8, 16 x ([22, 320] x [320, 16]) 30 -> 8.
#pragma once

namespace xb {

constexpr int HALF_BN = 64, HALF_BK = 64, HALF_PITCH = HALF_BK + 8, HALF_OPITCH = HALF_BN + 8;

template <int X4T>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  if constexpr (X4T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// c += a b as sums of 16 products, each added to c by an fp32 addition of its own: what the matrix instruction adds to an accumulator
// is cut off, not rounded, and a long chain of such sums drifts. The products of [16..512]-deep sums against 64 bits, rms relative to
// the result, before the result's rounding (fp32 FMAs; matrix instructions that accumulate): fp16 normal values 6.5e-8 (1.5e-7; 1.6e-7),
// positive ones 5.7e-8 (9.0e-8; 2.9e-7); bf16 4.5e-8 (5.6e-8; 1.0e-7) and 3.5e-8 (4.3e-8; 1.0e-7). Largest error: 0.3 to 0.7 of the FMAs'.
template <bool BF16>
__device__ __forceinline__ void mma_half(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += d[e];
}

// Blocks of `R` rows x 64 adjacent elements on their way to shared memory: warp w takes rows w, w + 8, ..., a lane elements 2 lane
// and the next. Zero past `rows` and `ext`. Where no more than 32 elements of a row are left, half a warp takes one (`narrow`; the
// upper 32 columns in shared memory are then not written).
template <int R>
struct HalfSlice {
  uint32_t v[R / 8];
  // ALL: every element is there (what most slices of a large product are, and half the instructions)
  template <int PASS, bool ALL, bool EVEN>
  __device__ __forceinline__ void fetch(const uint16_t* at, int64_t ld, int rows, bool one, bool two) {
    uint16_t lo[R / PASS], hi[R / PASS];
#pragma unroll
    for (int i = 0; i < R / PASS; ++i, at += PASS * ld) {
      const bool in = ALL || PASS * i < rows;
      if (EVEN) {
        v[i] = 0;
        if (ALL || (in && two)) v[i] = __ldg(reinterpret_cast<const uint32_t*>(at));
        else if (in && one) v[i] = __ldg(at);
      } else {
        lo[i] = hi[i] = 0;
        if (ALL || (in && one)) lo[i] = __ldg(at);
        if (ALL || (in && two)) hi[i] = __ldg(at + 1);
      }
    }
    if (!EVEN) {
#pragma unroll
      for (int i = 0; i < R / PASS; ++i) v[i] = (uint32_t)lo[i] | (uint32_t)hi[i] << 16;
    }
  }
  static __device__ __forceinline__ bool narrow(int c0, int ext) { return ext - c0 <= 32; }
  __device__ __forceinline__ void load(const uint16_t* base, int64_t ld, int row0, int rows, int c0, int ext, bool even) {
    const bool nar = narrow(c0, ext);
    const int lane = threadIdx.x & 31, w = nar ? threadIdx.x >> 4 : threadIdx.x >> 5, c = c0 + 2 * (nar ? lane & 15 : lane);
    const bool one = c < ext, two = c + 1 < ext, all = row0 + R <= rows && c0 + 64 <= ext;
    const uint16_t* at = base + (int64_t)(row0 + w) * ld + c;
    const int left = rows - row0 - w;
    if (even) {
      if (all) fetch<8, true, true>(at, ld, left, one, two);
      else if (nar) fetch<16, false, true>(at, ld, left, one, two);
      else fetch<8, false, true>(at, ld, left, one, two);
    } else {
      if (all) fetch<8, true, false>(at, ld, left, one, two);
      else if (nar) fetch<16, false, false>(at, ld, left, one, two);
      else fetch<8, false, false>(at, ld, left, one, two);
    }
  }
  __device__ __forceinline__ void store(uint16_t* s, int pitch, bool nar) const {
    if (nar) {
#pragma unroll
      for (int i = 0; i < R / 16; ++i)
        *reinterpret_cast<uint32_t*>(s + ((threadIdx.x >> 4) + 16 * i) * pitch + 2 * (threadIdx.x & 15)) = v[i];
    } else {
#pragma unroll
      for (int i = 0; i < R / 8; ++i)
        *reinterpret_cast<uint32_t*>(s + ((threadIdx.x >> 5) + 8 * i) * pitch + 2 * (threadIdx.x & 31)) = v[i];
    }
  }
};

// `finish` with one quotient for both activations that have one: with two, and their special cases, the loop over the outputs is so
// long that products without an activation pay for it ([30000, 500] x [500, 511] 153 us, 146; 8 x ([2254, 117] x [117, 144]) 22, 19)
__device__ __forceinline__ float half_finish(const SimtGemmParams& p, const Column& c, int b, int gm, int gn, float acc) {
  float v = p.alpha * acc;
  if (p.bias_kind == XB_BIAS_ROW)
    v += p.beta * c.bias;
  else if (p.bias_kind == XB_BIAS_FULL)
    v += p.beta * load_as_f32(p.bias, (int64_t)b * p.stride_bias + (int64_t)(gm / p.bias_group) * p.ldbias + gn, p.bias_dtype);
  if (p.epi.kind == XB_EPI_PRELU) return act_prelu(v, c.a);
  if (p.epi.kind == XB_EPI_NONE) return v;
  const bool dice = p.epi.kind == XB_EPI_DICE;
  const float s = 1.f / (1.f + __expf(dice ? -(v - c.b) * c.c : -v));
  return dice ? (1.f - s) * c.a * v + s * v : s;
}

// BM = 128: 4 x 2 warps of 32 x 32 outputs; BM = 64: 2 x 4 of 32 x 16.
template <bool BF16, int BM, bool TA, bool TB>
__global__ void __launch_bounds__(256, 2) gemm_half_kernel(const __grid_constant__ SimtGemmParams p, int a_even, int b_even) {
  constexpr int WN = BM == 128 ? 32 : 16, NF = WN / 8;
  constexpr int AHEAD = BM == 128 ? 1 : 2;                      // slices in registers: the small tile runs where few warps do
  constexpr int APITCH = TA ? BM + 8 : HALF_PITCH;              // A lies as [BM][64 k], transposed as [64 k][BM]
  constexpr int A_ELEMS = BM * HALF_PITCH, B_ELEMS = 64 * HALF_PITCH;
  constexpr int OUT_BYTES = BM * HALF_OPITCH * 4, RING_BYTES = (A_ELEMS + B_ELEMS) * 2;
  static_assert(!TA || HALF_BK * APITCH <= A_ELEMS, "both forms of A fit the same space");
  __shared__ __align__(16) uint8_t mem[OUT_BYTES > RING_BYTES ? OUT_BYTES : RING_BYTES];
  uint16_t* As = reinterpret_cast<uint16_t*>(mem);
  uint16_t* Bs = As + A_ELEMS;
  pdl_wait();
  const int b = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint16_t* A = reinterpret_cast<const uint16_t*>(p.A) + (int64_t)b * p.stride_a;
  const uint16_t* B = reinterpret_cast<const uint16_t*>(p.B) + (int64_t)b * p.stride_b;
  // neighbouring CTAs take the n tiles of one m tile: its rows come from L2 after the first
  const int mt = blockIdx.x / p.tiles_n, m0 = mt * BM, n0 = (int)(blockIdx.x - (unsigned)mt * p.tiles_n) * HALF_BN;
  const int nk = (p.K + HALF_BK - 1) / HALF_BK;

  struct Slices { HalfSlice<BM> a; HalfSlice<64> b; };           // (transposed: BM / 64 blocks of 64 rows of k)
  auto load = [&](Slices& s, int kb) {
    HalfSlice<BM>& sa = s.a;
    HalfSlice<64>& sb = s.b;
    const int k0 = kb * HALF_BK;
    if constexpr (TA) {
#pragma unroll
      for (int h = 0; h < BM / 64; ++h) {
        HalfSlice<64> t;
        t.load(A, p.lda, k0, p.K, m0 + 64 * h, p.M, a_even);
#pragma unroll
        for (int i = 0; i < 8; ++i) sa.v[8 * h + i] = t.v[i];
      }
    } else {
      sa.load(A, p.lda, m0, p.M, k0, p.K, a_even);
    }
    if constexpr (TB) sb.load(B, p.ldb, n0, p.N, k0, p.K, b_even);
    else sb.load(B, p.ldb, k0, p.K, n0, p.N, b_even);
  };
  auto store = [&](const Slices& s, int kb) {
    const int k0 = kb * HALF_BK;
    const HalfSlice<BM>& sa = s.a;
    const HalfSlice<64>& sb = s.b;
    if constexpr (TA) {
#pragma unroll
      for (int h = 0; h < BM / 64; ++h) {
        HalfSlice<64> t;
#pragma unroll
        for (int i = 0; i < 8; ++i) t.v[i] = sa.v[8 * h + i];
        t.store(As + 64 * h, APITCH, HalfSlice<64>::narrow(m0 + 64 * h, p.M));
      }
    } else {
      sa.store(As, APITCH, HalfSlice<BM>::narrow(k0, p.K));
    }
    sb.store(Bs, HALF_PITCH, HalfSlice<64>::narrow(TB ? k0 : n0, TB ? p.K : p.N));
  };

  const int wm = BM == 128 ? (warp >> 1) * 32 : (warp >> 2) * 32, wn = BM == 128 ? (warp & 1) * WN : (warp & 3) * WN;
  float acc[2][NF][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  // where this lane's row of a 16 x 16 piece lies; ldmatrix transposes what lies with k as its rows
  const int l8 = lane & 7, g1 = (lane >> 3) & 1, g2 = lane >> 4;
  const uint32_t as = (uint32_t)__cvta_generic_to_shared(As), bs = (uint32_t)__cvta_generic_to_shared(Bs);
  const uint32_t a_at = as + 2 * (TA ? (g2 * 8 + l8) * APITCH + wm + g1 * 8 : (wm + g1 * 8 + l8) * APITCH + g2 * 8);
  const uint32_t b_at = bs + 2 * (TB ? (wn + g2 * 8 + l8) * HALF_PITCH + g1 * 8 : (g1 * 8 + l8) * HALF_PITCH + wn + g2 * 8);

  Slices on_way[AHEAD];
#pragma unroll
  for (int u = 0; u < AHEAD; ++u)
    if (u < nk) load(on_way[u], u);
#pragma unroll 1
  for (int kb0 = 0; kb0 < nk; kb0 += AHEAD) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int kb = kb0 + u;
      if (kb >= nk) break;                                      // (the same for every thread)
      store(on_way[u], kb);
      __syncthreads();
      if (kb + AHEAD < nk) load(on_way[u], kb + AHEAD);
      const int depth = min(HALF_BK, p.K - kb * HALF_BK);       // (zeros up to a multiple of 16)
#pragma unroll
      for (int k = 0; k < HALF_BK; k += 16) {
        if (k >= depth) break;
        uint32_t af[2][4], bf[NF / 2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) ldmatrix4<TA>(af[i], a_at + 2 * (TA ? k * APITCH + 16 * i : 16 * i * APITCH + k));
#pragma unroll
        for (int j = 0; j < NF / 2; ++j) ldmatrix4<!TB>(bf[j], b_at + 2 * (TB ? 16 * j * HALF_PITCH + k : k * HALF_PITCH + 16 * j));
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < NF; ++j) mma_half<BF16>(acc[i][j], af[i], bf[j / 2][2 * (j & 1)], bf[j / 2][2 * (j & 1) + 1]);
      }
      __syncthreads();
    }
  }

  pdl_release();
  float* out = reinterpret_cast<float*>(mem);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(out + (wm + 16 * i + 8 * h + (lane >> 2)) * HALF_OPITCH + wn + 8 * j + 2 * (lane & 3)) =
            make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  __syncthreads();
  // a thread keeps its two columns and takes every eighth row (every sixteenth of up to 32 columns)
  const bool nar = p.N - n0 <= 32;
  const int cl = 2 * (nar ? lane & 15 : lane), gn = n0 + cl, step = nar ? 16 : 8;
  if (gn >= p.N) return;
  const bool two = gn + 1 < p.N;
  const Column c0 = column_of(p, b, gn), c1 = column_of(p, b, two ? gn + 1 : gn);
#pragma unroll 4
  for (int r = nar ? threadIdx.x >> 4 : warp; r < BM && m0 + r < p.M; r += step) {
    const float2 x = *reinterpret_cast<const float2*>(out + r * HALF_OPITCH + cl);
    const float v0 = half_finish(p, c0, b, m0 + r, gn, x.x), v1 = two ? half_finish(p, c1, b, m0 + r, gn + 1, x.y) : 0.f;
    const int64_t at = (int64_t)b * p.stride_y + (int64_t)(m0 + r) * p.ldy + gn;
    if (p.y_pairs && two) {
      uint32_t w;
      if (p.y_dtype == XB_BF16) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(v0, v1);
        w = *reinterpret_cast<const uint32_t*>(&t);
      } else {
        const __half2 t = __floats2half2_rn(v0, v1);
        w = *reinterpret_cast<const uint32_t*>(&t);
      }
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.Y) + at) = w;
    } else {
      store_from_f32(p.Y, at, p.y_dtype, v0);
      if (two) store_from_f32(p.Y, at + 1, p.y_dtype, v1);
    }
  }
}

template <bool BF16, int BM>
static void launch_half(const SimtGemmParams& p, dim3 grid, int a_even, int b_even, cudaStream_t s) {
  if (p.trans_a) {
    if (p.trans_b) launch_dependent(gemm_half_kernel<BF16, BM, true, true>, grid, 256, 0, s, p, a_even, b_even);
    else launch_dependent(gemm_half_kernel<BF16, BM, true, false>, grid, 256, 0, s, p, a_even, b_even);
  } else {
    if (p.trans_b) launch_dependent(gemm_half_kernel<BF16, BM, false, true>, grid, 256, 0, s, p, a_even, b_even);
    else launch_dependent(gemm_half_kernel<BF16, BM, false, false>, grid, 256, 0, s, p, a_even, b_even);
  }
}

// p as gemm_simt fills it. Tiles of 64 rows where those of 128 would not give every SM one.
static int gemm_half(SimtGemmParams& p, const xb_gemm_args& a, cudaStream_t s) {
  auto even = [](const void* ptr, int64_t ld, int64_t stride) {
    return (int)((reinterpret_cast<uintptr_t>(ptr) & 3) == 0 && ld % 2 == 0 && stride % 2 == 0);
  };
  const int a_even = even(a.A, a.lda, a.stride_a), b_even = even(a.B, a.ldb, a.stride_b);
  p.y_pairs = even(a.Y, a.ldy, a.stride_y);
  p.tiles_n = (a.N + HALF_BN - 1) / HALF_BN;
  const int64_t large = ((int64_t)a.M + 127) / 128 * p.tiles_n;
  const int bm = large * a.batch >= sm_count() ? 128 : 64;
  const int64_t tiles = ((int64_t)a.M + bm - 1) / bm * p.tiles_n;
  XB_REQUIRE(tiles < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gemm: %lld output tiles are too many for one call", (long long)tiles);
  const dim3 grid((unsigned)tiles, (unsigned)a.batch);
  if (a.ab_dtype == XB_BF16) {
    if (bm == 128) launch_half<true, 128>(p, grid, a_even, b_even, s);
    else launch_half<true, 64>(p, grid, a_even, b_even, s);
  } else {
    if (bm == 128) launch_half<false, 128>(p, grid, a_even, b_even, s);
    else launch_half<false, 64>(p, grid, a_even, b_even, s);
  }
  return check_launch("gemm_half_kernel");
}

}  // namespace xb
