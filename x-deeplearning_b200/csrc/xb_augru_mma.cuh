// AUGRU with the state in registers (included by xb_rnn.cu after xb_augru_tc.cuh, whose formulas and parameters it shares): for
// calls of few tiles, where the chain of a step is the time.
//
// A warp owns 16 candidates and all their columns, and both products of a step are warp-level MMAs (m16n8k16 / m16n8k8): their
// accumulators lie in registers as their A operand wants them, so h and r*h go from one product into the next without leaving
// the thread, and no thread waits for another one anywhere in the walk. The tcgen05 engine pays two tensor-memory round trips
// with their barriers a step, but its products cost the SM almost nothing, while these take the schedulers' slow path to the
// tensor cores: with one warp a scheduler a step is its chain (1180 cycles, 2110 there), with two the products bound it (1680).
// So this engine takes the calls that give every SM one CTA at the most: tcgen05 tiles share an SM in pairs beyond that.
// H = 36, 100 steps, us (tcgen05 engine): 200 candidates 65 (113), 4 x 1000 65 (114), 16 x 1000 90 (114); more CTAs than SMs,
// 19 x 1000: 178 (178), 74 x 1000: 356 (341).
//
// The terms of x_t are made once per CTA and chunk of steps and enter the products as they do in the tcgen05 engine: summed in
// fp32 in its order, rounded to fp16, and multiplied by a one in the first spare row of the last k chunk. With the same chunks of 16
// in k a state then has the same bits whichever engine the call's size picks. (As the fp32 start of the accumulators: 67 us instead
// of 65, 4 x 1000.) The recurrent weights stay in registers (H <= 36) or are read from shared memory as fragments. The state h stays
// in fp32; it is rounded to fp16 only as an MMA operand.
//
// Columns of the gate product in tiles of 8: the whole tiles of r, those of u, then one tile with what is left of both, so that
// no SFU work is spent on padding (H = 36: 9 tiles instead of 10); the u part of that tile moves to the lanes of its columns by
// one shuffle.
#pragma once

namespace xb {
namespace {

constexpr int AM_CHUNK = 128;             // steps whose request-side terms and scores are in shared memory at a time

template <int H>
struct AmGeom {
  static constexpr int HT = H / 8, W = H % 8;                   // whole tiles of 8 columns, columns left
  static constexpr int KT = HT + 1;                             // chunks of 8 in k
  static constexpr int NG = 2 * HT + 1, NC = HT + 1, NT = NG + NC;
  static constexpr int NPX = NT * 8;                            // request-side terms of a step, in tile order
  static constexpr int XP = KT * 8;                             // pitch of an x row
  static constexpr bool WREG = H <= 36;                         // recurrent weights in registers
  static_assert(W == 2 || W == 4, "two or four columns left over");
};
struct AmSmem { int wb, px, xs, att, total, n16, ap; };
template <int H>
__host__ __device__ inline AmSmem am_smem(int T, int warps) {
  using G = AmGeom<H>;
  AmSmem s;
  s.n16 = ((T < AM_CHUNK ? T : AM_CHUNK) + 15) / 16 * 16;
  s.ap = s.n16 + 2;                                             // an odd number of words: the rows of a warp on different banks
  int off = 0;
  s.wb = off; off += G::NT * G::KT * 128;                       // fragments of the recurrent weights: [tile][k chunk][lane]
  s.px = off; off += (s.n16 + 1) * G::NPX * 2;                  // (one row more: the last step requests a next one)
  s.xs = off; off += s.n16 * G::XP * 2;
  s.att = off; off += warps * 16 * s.ap * 2;
  s.total = (off + 15) / 16 * 16;
  return s;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
// acc += A W for one tile of 8 columns: a[chunk][row half], b(chunk) the tile's weight fragment
template <int KT, typename B>
__device__ __forceinline__ void am_product(float (&acc)[4], const uint32_t (&a)[KT][2], B b) {
#pragma unroll
  for (int k = 0; k + 1 < KT; k += 2) mma_16816(acc, a[k][0], a[k][1], a[k + 1][0], a[k + 1][1], b(k), b(k + 1));
  if constexpr (KT & 1) mma_1688(acc, a[KT - 1][0], a[KT - 1][1], b(KT - 1));
}

// column of Wg (r first, then u) or Wc that position n of tile j stands for, -1: padding
template <int H>
__device__ __forceinline__ int am_column(int j, int n) {
  using G = AmGeom<H>;
  if (j < G::HT) return j * 8 + n;
  if (j < 2 * G::HT) return H + (j - G::HT) * 8 + n;
  if (j == 2 * G::HT) return n < G::W ? G::HT * 8 + n : n < 2 * G::W ? H + G::HT * 8 + n - G::W : -1;
  const int c = (j - G::NG) * 8 + n;
  return c < H ? c : -1;
}
// rows k0 and k0 + 1 of the h part of a weight column, as one fragment word
template <int H>
__device__ __forceinline__ uint32_t am_weights(const AuParams& p, int j, int col, int k0) {
  const bool gate = j < AmGeom<H>::NG;
  const __half* W = gate ? p.Wg : p.Wc;
  const int ld = gate ? 2 * H : H;
  const __half zero = __float2half(0.f);
  const __half lo = col >= 0 && k0 < H ? W[(H + k0) * ld + col] : zero, hi = col >= 0 && k0 + 1 < H ? W[(H + k0 + 1) * ld + col] : zero;
  return h2_bits(__halves2half2(lo, hi));
}

template <int H>
__global__ void __launch_bounds__(256, 1) augru_mma_kernel(const __grid_constant__ AuParams p) {
  using G = AmGeom<H>;
  constexpr int HT = G::HT, KT = G::KT, NG = G::NG, NC = G::NC, NT = G::NT, NPX = G::NPX;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, q = lane & 3;                        // row of the warp's 16 (and g + 8), column pair of a tile
  const AmSmem S = am_smem<H>(p.T, warps);
  uint32_t* wb = reinterpret_cast<uint32_t*>(smem + S.wb);
  __half* px = reinterpret_cast<__half*>(smem + S.px);
  __half* xs = reinterpret_cast<__half*>(smem + S.xs);
  __half* atts = reinterpret_cast<__half*>(smem + S.att);
  const int r = blockIdx.x / p.tiles_per_req, first = (blockIdx.x - r * p.tiles_per_req) * warps * 16;
  const int rows = min(warps * 16, p.n_cand - first), T = p.T;
  const __half zero = __float2half(0.f);
  const bool slot = q == G::W / 2;                              // this lane has the first spare row of the last k chunk: a one in A
  const uint32_t one = slot ? 0x3C00u : 0u;

#pragma unroll 4
  for (int i = tid; i < NT * KT * 32; i += blockDim.x) {
    const int l = i & 31, k = (i >> 5) % KT, j = (i >> 5) / KT;
    wb[i] = am_weights<H>(p, j, am_column<H>(j, l >> 2), 8 * k + 2 * (l & 3));
  }

  float h[NC][4];
  uint32_t hp[KT][2];                                           // h as the A operand
#pragma unroll
  for (int j = 0; j < NC; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e) h[j][e] = 0.f;
    hp[j][0] = hp[j][1] = j == HT ? one : 0u;
  }
  uint32_t wr[G::WREG ? NT : 1][KT];
  const __half* xr = p.x + (int64_t)r * T * H;
  const __half* ar = p.att + ((int64_t)r * p.n_cand + first) * T;
  const bool a8 = T % 4 == 0 && (reinterpret_cast<uintptr_t>(p.att) & 7) == 0;
  const bool x4 = (reinterpret_cast<uintptr_t>(p.x) & 3) == 0;  // H is even

  for (int t0 = 0; t0 < T; t0 += AM_CHUNK) {
    const int n = min(AM_CHUNK, T - t0), n16 = (n + 15) / 16 * 16;
    if (t0 > 0) __syncthreads();                                // the last chunk has been walked
    // ---- the chunk's inputs and scores
#pragma unroll 4
    for (int i = tid; i < n16 * (KT * 4); i += blockDim.x) {
      const int t = i / (KT * 4), k = (i - t * (KT * 4)) * 2;
      const __half* src = xr + (int64_t)(t0 + t) * H + k;
      uint32_t v = 0u;
      if (t < n && k < H) v = x4 ? *reinterpret_cast<const uint32_t*>(src) : h2_bits(__halves2half2(src[0], src[1]));
      *reinterpret_cast<uint32_t*>(xs + t * G::XP + k) = v;
    }
    if (a8) {
      const int n4 = n / 4;                                     // n is T, AM_CHUNK or their remainder: a multiple of 4
#pragma unroll 4
      for (int i = tid; i < warps * 16 * n4; i += blockDim.x) {
        const int row = i / n4, c = (i - row * n4) * 4;
        uint2 v = make_uint2(0u, 0u);
        if (row < rows) v = *reinterpret_cast<const uint2*>(ar + (int64_t)row * T + t0 + c);
        uint32_t* dst = reinterpret_cast<uint32_t*>(atts + row * S.ap + c);
        dst[0] = v.x; dst[1] = v.y;
      }
    } else {
#pragma unroll 4
      for (int i = tid; i < warps * 16 * n; i += blockDim.x) {
        const int row = i / n, c = i - row * n;
        atts[row * S.ap + c] = row < rows ? ar[(int64_t)row * T + t0 + c] : zero;
      }
    }
    __syncthreads();
    // ---- request-side terms x_t Wx + b: a column a thread, its weights in registers, four steps at a time
    for (int i = tid & 127; i < NPX; i += 128) {
      const int j = i >> 3, c = am_column<H>(j, i & 7);
      const bool gate = j < NG;
      const __half* W = gate ? p.Wg : p.Wc;
      const int ld = gate ? 2 * H : H;
      float w[H];
#pragma unroll
      for (int k = 0; k < H; ++k) w[k] = c >= 0 ? __half2float(W[k * ld + c]) : 0.f;
      const float bias = c >= 0 ? __half2float((gate ? p.bg : p.bc)[c]) : 0.f;
      const int share = tid >> 7, shares = blockDim.x >> 7;
      for (int t = 4 * share; t < n; t += 4 * shares) {
        float v[4] = {bias, bias, bias, bias};
#pragma unroll
        for (int k = 0; k < H; k += 2) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {                         // (rows up to a multiple of 16 are there, zero past the last step)
            const float2 xv = __half22float2(*reinterpret_cast<const __half2*>(xs + (t + e) * G::XP + k));
            v[e] = fmaf(xv.y, w[k + 1], fmaf(xv.x, w[k], v[e]));
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) px[(t + e) * NPX + i] = __float2half_rn(v[e]);
      }
    }
    if constexpr (G::WREG) {
      if (t0 == 0) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int k = 0; k < KT; ++k) wr[j][k] = wb[(j * KT + k) * 32 + lane];
      }
    }
    __syncthreads();

    // ---- the steps
    const uint16_t* pxl = reinterpret_cast<const uint16_t*>(px) + g;
    const __half* al = atts + (warp * 16 + g) * S.ap;
    float acc[NT][4];
    uint32_t last[NT];                                          // fragments of the last k chunk: weights, in the slot's lanes the step's term
    auto start = [&](int j, int t) {
      if (slot) last[j] = pxl[t * NPX + j * 8];
    };
    auto weight = [&](int j, int k) {
      if (k == KT - 1) return last[j];
      if constexpr (G::WREG) return wr[j][k];
      else return wb[(j * KT + k) * 32 + lane];
    };
    // sigmoid(z) = 1/2 + 1/2 tanh(z/2), two columns per SFU instruction
    auto sigm2 = [](float a, float b) {
      const __half2 z = __floats2half2_rn(0.5f * a, 0.5f * b);
      const __half2 th = bits_h2(umma::tanh_f16x2(h2_bits(z)));
      return h2_bits(__hfma2(th, __floats2half2_rn(0.5f, 0.5f), __floats2half2_rn(0.5f, 0.5f)));
    };
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      last[j] = wb[(j * KT + KT - 1) * 32 + lane];
      start(j, 0);
    }
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
      const float om[2] = {1.f - __half2float(al[t]), 1.f - __half2float(al[8 * S.ap + t])};
      // gates: r's tiles first, r*h is what the candidate product waits for
      auto product = [&](int j, const uint32_t (&a)[KT][2]) {
        acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
        am_product<KT>(acc[j], a, [&](int k) { return weight(j, k); });
      };
      auto gate = [&](int j) { product(j, hp); };
#pragma unroll
      for (int j = 0; j < HT; ++j) gate(j);
      gate(2 * HT);
#pragma unroll
      for (int j = HT; j < 2 * HT; ++j) gate(j);
      uint32_t rh[KT][2], u[NC][2];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int tile = j < HT ? j : 2 * HT;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t s = sigm2(acc[tile][2 * e], acc[tile][2 * e + 1]);
          const float2 rf = __half22float2(bits_h2(s));
          rh[j][e] = h2_bits(__floats2half2_rn(rf.x * h[j][2 * e], rf.y * h[j][2 * e + 1]));   // (h is zero past column H)
          if (j == HT && slot) rh[j][e] = one;
          if (j == HT) {
            const uint32_t moved = __shfl_down_sync(0xffffffffu, s, G::W / 2);
            u[HT][e] = q < G::W / 2 ? moved : 0u;               // (padding columns take nothing from another candidate)
          }
        }
        start(tile, t + 1);
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) product(NG + j, rh);
#pragma unroll
      for (int j = 0; j < HT; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) u[j][e] = sigm2(acc[HT + j][2 * e], acc[HT + j][2 * e + 1]);
        start(HT + j, t + 1);
      }
      // candidate and blend
#pragma unroll
      for (int j = 0; j < NC; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const __half2 z = __floats2half2_rn(acc[NG + j][2 * e], acc[NG + j][2 * e + 1]);
          const float2 c = __half22float2(bits_h2(umma::tanh_f16x2(h2_bits(z))));
          const float2 uf = __half22float2(bits_h2(u[j][e]));
          const float u0 = om[e] * uf.x, u1 = om[e] * uf.y;
          h[j][2 * e] = u0 * h[j][2 * e] + (1.f - u0) * c.x;
          h[j][2 * e + 1] = u1 * h[j][2 * e + 1] + (1.f - u1) * c.y;
          hp[j][e] = h2_bits(__floats2half2_rn(h[j][2 * e], h[j][2 * e + 1]));
          if (j == HT && slot) hp[j][e] = one;
        }
        start(NG + j, t + 1);
      }
    }
  }
  pdl_release();
  const int row = warp * 16 + g;
  __half* out = p.y + ((int64_t)r * p.n_cand + first + row) * H + 2 * q;       // H is even: 4-byte aligned (y is)
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    if (j * 8 + 2 * q >= H) continue;
    if (row < rows) *reinterpret_cast<uint32_t*>(out + j * 8) = hp[j][0];
    if (row + 8 < rows) *reinterpret_cast<uint32_t*>(out + (int64_t)8 * H + j * 8) = hp[j][1];
  }
}

// 128 candidates a CTA: one CTA an SM. (The widths are those of the tcgen05 engine, all of them H % 8 == 2 or 4.)
bool augru_mma_wanted(const AuParams& p) { return (int64_t)p.requests * ((p.n_cand + 127) / 128) <= sm_count(); }

template <int H>
int launch_augru_mma_h(AuParams p, cudaStream_t stream) {
  static PerDeviceOnce attr;                          // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr, am_smem<H>(AM_CHUNK, 8).total, (const void*)augru_mma_kernel<H>);
  // eight warps of 16 candidates; four where every SM then still has one CTA at the most, and its schedulers one warp each
  const int warps = (int64_t)p.requests * ((p.n_cand + 63) / 64) <= sm_count() ? 4 : 8;
  p.tiles_per_req = (p.n_cand + warps * 16 - 1) / (warps * 16);
  const int64_t blocks = (int64_t)p.requests * p.tiles_per_req;
  launch_dependent(augru_mma_kernel<H>, (unsigned)blocks, warps * 32, am_smem<H>(p.T, warps).total, stream, p);
  return check_launch("augru_mma_kernel");
}

int launch_augru_mma(const AuParams& p, cudaStream_t stream) {
  // one instantiation per eligible H
  switch (p.H) {
#define XB_AU_CASE(h) case h: return launch_augru_mma_h<h>(p, stream)
    XB_AU_CASE(4); XB_AU_CASE(10); XB_AU_CASE(12); XB_AU_CASE(18); XB_AU_CASE(20); XB_AU_CASE(26); XB_AU_CASE(28);
    XB_AU_CASE(34); XB_AU_CASE(36); XB_AU_CASE(42); XB_AU_CASE(44); XB_AU_CASE(50); XB_AU_CASE(52); XB_AU_CASE(58);
    XB_AU_CASE(60);
#undef XB_AU_CASE
    default: return fail(XB_ERR_UNSUPPORTED, "xb_augru_shared: H = %d", p.H);
  }
}

}  // namespace
}  // namespace xb
