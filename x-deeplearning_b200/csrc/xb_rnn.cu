// GRU and attention-gated GRU (AUGRU) over short behaviour sequences.
//
// One CTA owns one sequence and walks its T steps, so a sequence never leaves
// its SM and needs no inter-CTA synchronisation (the reference CUDA GRU spins on
// global atomics between blocks, blaze/blaze/operator/op/gru_op.cu:73-85; nothing
// here waits on another CTA). Latency-bound by design: throughput comes from
// batch-many independent CTAs.
#include <algorithm>
#include <cstring>

#include "xb_common.cuh"
#include "xb_umma.cuh"

namespace xb {
namespace {

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

__device__ __forceinline__ float sigm(float v) { return 1.f / (1.f + expf(-v)); }

}  // namespace
}  // namespace xb

#include "xb_augru_tc.cuh"
#include "xb_augru_mma.cuh"

namespace xb {
namespace {

// x [B,T,H], y [B,T,H]; i2h, h2h [H,3H] (gate order r, z, candidate); biases [3H].
// Follows GRUKernel, blaze/blaze/operator/op/gru_op.cc:33-93: leading steps whose first H
// input pre-activations (before the bias) are all zero emit zeros and leave h at zero.
//
// What bounds it is the chain h(t) -> h(t+1), in which every instruction waits for the one before; everything else is kept off
// it. The input products of up to GRU_CHUNK steps are made first (they do not depend on h). Then a thread owns one of the 3H
// gate columns, its recurrent weights in registers, and a step is: read h as broadcast 16-byte vectors, eight chains of FMAs,
// the reset and update threads evaluate their gates and leave them in shared memory, the candidate threads the candidate and the
// new h. Two barriers a step, but no shuffles, and each scheduler has one warp (H = 36).
// The data type is that of the arrays: state, sums and gates (expf, tanhf, a division) are fp32 for either.
// 16 sequences of 100 steps, H = 36: 42 us fp16, 38 fp32; 61 and 57 with four lanes a unit, three shuffles and one barrier a step.
// The chains add up as those lanes did, so the results are the same (four chains, one a component of the vectors: 41.5 and 38).
// 16 of H = 64 57 and 53. (The register bound lets the compiler have every h vector of a step on its way at once: at 128
// registers, which it picks otherwise, 56 us; calls of many sequences have other bounds, see launch_gru_nv.)
constexpr int GRU_CHUNK = 64;
__host__ __device__ constexpr int gru_hp(int nv) { return 16 * nv; }          // h and x rows padded with zeros

template <typename T, int NV, int BLOCKS>
__global__ void __launch_bounds__((48 * NV + 31) / 32 * 32, BLOCKS) gru_kernel(const T* x, T* y, int steps, int H,
                                                                       const T* __restrict__ i2h, const T* __restrict__ h2h,
                                                                       const T* __restrict__ bi, const T* __restrict__ bh) {
  pdl_wait();
  constexpr int HP = gru_hp(NV);
  extern __shared__ __align__(16) float gru_sm[];
  float* xs = gru_sm;                              // [GRU_CHUNK][HP]
  float* pre = xs + GRU_CHUNK * HP;                // [GRU_CHUNK][3H]: input products with their bias
  __shared__ __align__(16) float hbuf[HP];
  __shared__ float gates[2 * HP];
  __shared__ int first_s;                          // first step of the chunk with a non-zero among its first H input products
  const int tid = threadIdx.x, G = 3 * H;
  const bool col = tid < G;                        // gate column tid: r, z, candidate
  const int u = tid - 2 * H;                       // candidate threads: their unit
  const int64_t b = blockIdx.x;
  float wi[HP], wh[HP];                            // column tid of i2h and of h2h
#pragma unroll
  for (int k = 0; k < HP; ++k) {
    wi[k] = (k < H && col) ? to_f32<T>(i2h[k * G + tid]) : 0.f;
    wh[k] = (k < H && col) ? to_f32<T>(h2h[k * G + tid]) : 0.f;
  }
  const float bij = col ? to_f32<T>(bi[tid]) : 0.f, bhj = col ? to_f32<T>(bh[tid]) : 0.f;
  for (int i = tid; i < HP; i += blockDim.x) hbuf[i] = 0.f;
  bool started = false;                            // the same for every thread
  float h = 0.f;
  for (int t0 = 0; t0 < steps; t0 += GRU_CHUNK) {
    const int n = min(GRU_CHUNK, steps - t0);
    __syncthreads();                               // the last chunk's rows have been used
    const T* xb = x + (b * steps + t0) * H;
    for (int i0 = tid; i0 < n * HP; i0 += 8 * blockDim.x) {       // eight loads in flight
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = i0 + e * (int)blockDim.x, t = i / HP, k = i - t * HP;
        v[e] = i < n * HP && k < H ? to_f32<T>(xb[t * H + k]) : 0.f;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = i0 + e * (int)blockDim.x;
        if (i < n * HP) xs[i] = v[e];
      }
    }
    if (tid == 0) first_s = n;
    __syncthreads();
    if (col) {
      int first = n;
      for (int t = 0; t < n; t += 4) {                            // four independent chains (rows past n are not kept)
        float q[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < HP; k += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 v = *reinterpret_cast<const float4*>(xs + (t + e) * HP + k);
            q[e] = fmaf(v.x, wi[k], q[e]); q[e] = fmaf(v.y, wi[k + 1], q[e]); q[e] = fmaf(v.z, wi[k + 2], q[e]); q[e] = fmaf(v.w, wi[k + 3], q[e]);
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          first = q[e] != 0.f ? min(first, t + e) : first;
          if (t + e < n) pre[(t + e) * G + tid] = q[e] + bij;
        }
      }
      if (!started && tid < H) atomicMin(&first_s, first);        // (steps past n are no less than n)
    }
    __syncthreads();
    if (t0 + n >= steps) pdl_release();            // (not in the steps: they are the chain)
    int t = 0;
    T* yt = y + (b * steps + t0) * H + u;
    if (!started) {                                // steps before the list begins: zeros, and a state of zero
      const int begin = first_s;
      for (; t < begin; ++t, yt += H)
        if (col && u >= 0) *yt = from_f32<T>(0.f);
      started = begin < n;
    }
    float pre_next = col && t < n ? pre[t * G + tid] : 0.f;
    for (; t < n; ++t, yt += H) {
      const float pre_j = pre_next;
      if (col && t + 1 < n) pre_next = pre[(t + 1) * G + tid];
      float a[4][2] = {};                          // quarter l of the units: 4 l .. 4 l + 3 of every 16
#pragma unroll
      for (int k = 0; k < HP; k += 4) {
        const float4 v = *reinterpret_cast<const float4*>(hbuf + k);
        float (&q)[2] = a[k / 4 % 4];
        q[0] = fmaf(v.x, wh[k], q[0]); q[1] = fmaf(v.y, wh[k + 1], q[1]); q[0] = fmaf(v.z, wh[k + 2], q[0]); q[1] = fmaf(v.w, wh[k + 3], q[1]);
      }
      const float sum = (((a[0][0] + a[0][1]) + (a[1][0] + a[1][1])) + ((a[2][0] + a[2][1]) + (a[3][0] + a[3][1]))) + bhj;
      if (tid < 2 * H) gates[tid] = sigm(pre_j + sum);
      __syncthreads();                             // the gates are there, and everyone has read h
      if (col && u >= 0) {
        const float r = gates[u], z = gates[H + u];
        const float c = tanhf(pre_j + r * sum);
        h = c + z * (h - c);
        hbuf[u] = h;
        *yt = from_f32<T>(h);
      }
      __syncthreads();
    }
  }
}

// AUGRU after VecAttGRUCell.call (xdl-algorithm-solution/DIEN/script/utils.py:139-207):
// [r|u] = sigmoid([x,h] Wg + bg); c = tanh([x, r*h] Wc + bc); u' = (1 - a_t) u; h' = u' h + (1 - u') c.
// Wg [2H, 2H] (rows x then h; columns r then u), Wc [2H, H]; att [B, T].
__global__ void augru_kernel(const void* x, const void* att, void* y, int T, int H, const void* Wg_, const void* bg_,
                             const void* Wc_, const void* bc_, int dt) {
  pdl_wait();
  extern __shared__ float sm[];
  float* Wg = sm;                     // [2H][2H]
  float* Wc = Wg + 4 * H * H;         // [2H][H]
  float* h = Wc + 2 * H * H;          // [H]
  float* xs = h + H;                  // [H]
  float* g = xs + H;                  // [2H]
  float* rh = g + 2 * H;              // [H]
  const int j = threadIdx.x, G = 2 * H;
  const int64_t b = blockIdx.x;
  for (int i = j; i < 4 * H * H; i += blockDim.x) Wg[i] = load_as_f32(Wg_, i, dt);
  for (int i = j; i < 2 * H * H; i += blockDim.x) Wc[i] = load_as_f32(Wc_, i, dt);
  if (j < H) h[j] = 0.f;
  const float bgj = j < G ? load_as_f32(bg_, j, dt) : 0.f, bcj = j < H ? load_as_f32(bc_, j, dt) : 0.f;
  __syncthreads();
  for (int t = 0; t < T; ++t) {
    const int64_t base = (b * T + t) * H;
    if (j < H) xs[j] = load_as_f32(x, base + j, dt);
    __syncthreads();
    if (j < G) {
      float s = bgj;
      for (int k = 0; k < H; ++k) s = fmaf(xs[k], Wg[k * G + j], s);
      for (int k = 0; k < H; ++k) s = fmaf(h[k], Wg[(H + k) * G + j], s);
      g[j] = sigm(s);
    }
    __syncthreads();
    if (j < H) rh[j] = g[j] * h[j];
    __syncthreads();
    float out = 0.f;
    if (j < H) {
      float s = bcj;
      for (int k = 0; k < H; ++k) s = fmaf(xs[k], Wc[k * H + j], s);
      for (int k = 0; k < H; ++k) s = fmaf(rh[k], Wc[(H + k) * H + j], s);
      const float a = load_as_f32(att, b * T + t, dt);
      const float u = (1.f - a) * g[H + j];
      out = u * h[j] + (1.f - u) * tanhf(s);
      store_from_f32(y, base + j, dt, out);
    }
    __syncthreads();
    if (j < H) h[j] = out;
  }
}

// AUGRU over a request's shared sequence in fp32, for widths the tensor-core engine does not take (and on request): x is
// [requests, T, H], att [requests * n_cand, T], only the final states y [requests * n_cand, H] are written.
// A CTA owns AS_CAND candidates of one request. The terms of x_t are the same for all of them: each chunk of steps they
// are made once, a gate column per thread. A candidate is four lanes per unit with their quarter of the unit's three
// recurrent columns in registers, and two barriers of its own threads a step: r*h, then h.
// 4 requests of 1000 candidates, 100 steps, H = 32: 418 us,
// 973 with a block per candidate and the weights in shared memory
constexpr int AS_CAND = 4, AS_CHUNK = 32;
template <int NV>
__global__ void __launch_bounds__(AS_CAND * 64 * NV > 1024 ? 1024 : AS_CAND * 64 * NV)
augru_shared_kernel(const __half* __restrict__ x, const __half* __restrict__ att, __half* __restrict__ y, int n_cand, int steps, int H,
                    const __half* __restrict__ Wg, const __half* __restrict__ bg, const __half* __restrict__ Wc,
                    const __half* __restrict__ bc, int cands, int group_threads, int blocks_per_req) {
  constexpr int HP = gru_hp(NV);
  extern __shared__ __align__(16) float as_sm[];
  float* xs = as_sm;                                           // [AS_CHUNK][HP]
  float* px = xs + AS_CHUNK * HP;                              // [AS_CHUNK][3H]: x_t Wg_x + bg (r, u), x_t Wc_x + bc
  __shared__ __align__(16) float hbuf[AS_CAND][2][HP];
  __shared__ __align__(16) float rhbuf[AS_CAND][HP];
  pdl_wait();
  const int tid = threadIdx.x, G = 3 * H;
  const int r = blockIdx.x / blocks_per_req, cand = tid / group_threads, gt = tid - cand * group_threads;
  const int n = (blockIdx.x - r * blocks_per_req) * cands + cand;
  const int u = gt >> 2, l = gt & 3;
  const bool unit = u < H && n < n_cand;
  float wr[4 * NV], wu[4 * NV], wc[4 * NV];
#pragma unroll
  for (int i = 0; i < 4 * NV; ++i) {
    const int k = 4 * (4 * (i >> 2) + l) + (i & 3);
    const bool in = u < H && k < H;
    wr[i] = in ? __half2float(Wg[(H + k) * 2 * H + u]) : 0.f;
    wu[i] = in ? __half2float(Wg[(H + k) * 2 * H + H + u]) : 0.f;
    wc[i] = in ? __half2float(Wc[(H + k) * H + u]) : 0.f;
  }
  for (int i = gt; i < 2 * HP; i += group_threads) (&hbuf[cand][0][0])[i] = 0.f;
  for (int i = gt; i < HP; i += group_threads) rhbuf[cand][i] = 0.f;
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(cand + 1), "r"(group_threads) : "memory"); };
  const __half* arow = att + ((int64_t)r * n_cand + min(n, n_cand - 1)) * steps;
  float h = 0.f;
  for (int t0 = 0; t0 < steps; t0 += AS_CHUNK) {
    const int m = min(AS_CHUNK, steps - t0);
    __syncthreads();
    for (int i = tid; i < m * HP; i += blockDim.x) {
      const int t = i / HP, k = i - t * HP;
      xs[i] = k < H ? __half2float(x[((int64_t)r * steps + t0 + t) * H + k]) : 0.f;
    }
    __syncthreads();
    for (int idx = tid; idx < m * G; idx += blockDim.x) {
      const int t = idx / G, j = idx - t * G;
      const bool gate = j < 2 * H;
      const __half* W = gate ? Wg + j : Wc + j - 2 * H;
      const int ld = gate ? 2 * H : H;
      float s = __half2float(gate ? bg[j] : bc[j - 2 * H]);
#pragma unroll 8
      for (int k = 0; k < H; ++k) s = fmaf(xs[t * HP + k], __half2float(__ldg(W + k * ld)), s);
      px[idx] = s;
    }
    __syncthreads();
    if (t0 + m >= steps) pdl_release();
    for (int t = 0; t < m; ++t) {
      const float a = __half2float(__ldg(arow + t0 + t));
      float pr = 0.f, pu = 0.f, pc = 0.f;
      if (unit) { pr = px[t * G + u]; pu = px[t * G + H + u]; pc = px[t * G + 2 * H + u]; }
      const float4* hv = reinterpret_cast<const float4*>(hbuf[cand][t & 1]);
      float ar = 0.f, au = 0.f, ac = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float4 v = hv[4 * i + l];
        ar = fmaf(v.x, wr[4 * i], ar); ar = fmaf(v.y, wr[4 * i + 1], ar); ar = fmaf(v.z, wr[4 * i + 2], ar); ar = fmaf(v.w, wr[4 * i + 3], ar);
        au = fmaf(v.x, wu[4 * i], au); au = fmaf(v.y, wu[4 * i + 1], au); au = fmaf(v.z, wu[4 * i + 2], au); au = fmaf(v.w, wu[4 * i + 3], au);
      }
      ar += __shfl_xor_sync(0xffffffffu, ar, 1); ar += __shfl_xor_sync(0xffffffffu, ar, 2);
      au += __shfl_xor_sync(0xffffffffu, au, 1); au += __shfl_xor_sync(0xffffffffu, au, 2);
      const float rg = sigm(pr + ar);
      if (unit && l == 0) rhbuf[cand][u] = rg * h;
      group_sync();
      const float ug = (1.f - a) * sigm(pu + au);
      const float4* rv = reinterpret_cast<const float4*>(rhbuf[cand]);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float4 v = rv[4 * i + l];
        ac = fmaf(v.x, wc[4 * i], ac); ac = fmaf(v.y, wc[4 * i + 1], ac); ac = fmaf(v.z, wc[4 * i + 2], ac); ac = fmaf(v.w, wc[4 * i + 3], ac);
      }
      ac += __shfl_xor_sync(0xffffffffu, ac, 1); ac += __shfl_xor_sync(0xffffffffu, ac, 2);
      h = ug * h + (1.f - ug) * tanhf(pc + ac);
      if (unit && l == 0) hbuf[cand][(t + 1) & 1][u] = h;
      group_sync();
    }
  }
  if (unit && l == 0) y[((int64_t)r * n_cand + n) * H + u] = __float2half_rn(h);
}

template <int NV>
int launch_augru_shared(const AuParams& p, cudaStream_t s) {
  const int gt = (4 * p.H + 31) / 32 * 32, cands = std::min(AS_CAND, 1024 / gt), bpr = (p.n_cand + cands - 1) / cands;
  XB_REQUIRE((int64_t)p.requests * bpr < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_augru_shared: batch too large");
  const size_t smem = sizeof(float) * AS_CHUNK * (size_t)(gru_hp(NV) + 3 * p.H);
  launch_dependent(augru_shared_kernel<NV>, (unsigned)(p.requests * bpr), cands * gt, smem, s, p.x, p.att, p.y, p.n_cand, p.T, p.H, p.Wg,
                   p.bg, p.Wc, p.bc, cands, gt, bpr);
  return check_launch("augru_shared_kernel");
}

template <typename T, int NV, int BLOCKS>
int launch_gru_blocks(const T* x, T* y, int64_t batch, int steps, int H, const T* i2h, const T* h2h, const T* bi, const T* bh,
                      cudaStream_t s) {
  const size_t smem = sizeof(float) * GRU_CHUNK * (size_t)(gru_hp(NV) + 3 * H);
  static PerDeviceOnce attr;                       // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr, sizeof(float) * GRU_CHUNK * 4 * gru_hp(NV), (const void*)gru_kernel<T, NV, BLOCKS>);
  launch_dependent(gru_kernel<T, NV, BLOCKS>, (unsigned)batch, (3 * H + 31) / 32 * 32, smem, s, x, y, steps, H, i2h, h2h, bi, bh);
  return check_launch("gru_kernel");
}
template <typename T, int NV>
int launch_gru_nv(const T* x, T* y, int64_t batch, int steps, int H, const T* i2h, const T* h2h, const T* bi, const T* bh,
                  cudaStream_t s) {
  // More sequences than are resident with all the registers that a step would like: a bound that lets more of them in. A quarter of
  // the register file holds three warps of 146 registers (NV = 2), two of 174 and 206. us of 40 steps in fp32, all registers and
  // bounded: 600 of H = 32 31, 23 (445: 20, 23); 300 of H = 36 37, 33 (200: 22, 26); 200 of H = 45 39, 28, 2000 269, 151;
  // 200 of H = 64 45, 31.
  constexpr int BLOCKS = NV == 2 ? 5 : NV == 3 ? 3 : NV == 4 ? 2 : 1;
  const int fit = NV == 2 ? 4 : NV == 3 && 3 * H <= 128 ? 2 : 1;
  if (BLOCKS > 1 && batch > (int64_t)fit * sm_count()) return launch_gru_blocks<T, NV, BLOCKS>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
  return launch_gru_blocks<T, NV, 1>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
}
template <typename T>
int launch_gru(const T* x, T* y, int64_t batch, int steps, int H, const T* i2h, const T* h2h, const T* bi, const T* bh,
               cudaStream_t s) {
  switch ((H + 15) / 16) {
    case 1: return launch_gru_nv<T, 1>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
    case 2: return launch_gru_nv<T, 2>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
    case 3: return launch_gru_nv<T, 3>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
    default: return launch_gru_nv<T, 4>(x, y, batch, steps, H, i2h, h2h, bi, bh, s);
  }
}

}  // namespace
}  // namespace xb

namespace xb {
int rnn_status(int* out) { return umma::read_status_word(out); }
int rnn_clear_status() { return umma::clear_status_word(); }
int rnn_set_status_mirror(int* p) { return umma::set_status_mirror(p); }
}  // namespace xb

using namespace xb;

extern "C" int xb_gru(const void* x, void* y, int64_t batch, int32_t T, int32_t H, const void* i2h, const void* h2h,
                      const void* i2h_bias, const void* h2h_bias, int32_t dtype, xb_stream_t s) {
  XB_REQUIRE(x && y && i2h && h2h && i2h_bias && h2h_bias, XB_ERR_ARG, "xb_gru: null tensor");
  XB_REQUIRE(batch >= 0 && T >= 0 && H >= 1, XB_ERR_ARG, "xb_gru: bad sizes");
  XB_REQUIRE(H <= 64, XB_ERR_LIMIT, "xb_gru: hidden size %d, at most 64 (weights are kept in registers)", H);
  XB_REQUIRE(dtype == XB_F32 || dtype == XB_F16, XB_ERR_UNSUPPORTED, "xb_gru: dtype %d", dtype);
  XB_REQUIRE(batch < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_gru: batch too large");
  if (batch == 0 || T == 0) return 0;
  const cudaStream_t stream = (cudaStream_t)s;
  if (dtype == XB_F32)
    return launch_gru((const float*)x, (float*)y, batch, T, H, (const float*)i2h, (const float*)h2h, (const float*)i2h_bias,
                      (const float*)h2h_bias, stream);
  return launch_gru((const __half*)x, (__half*)y, batch, T, H, (const __half*)i2h, (const __half*)h2h, (const __half*)i2h_bias,
                    (const __half*)h2h_bias, stream);
}

extern "C" int xb_augru(const void* x, const void* att, void* y, int64_t batch, int32_t T, int32_t H, const void* Wg,
                        const void* bg, const void* Wc, const void* bc, int32_t dtype, xb_stream_t s) {
  XB_REQUIRE(x && att && y && Wg && bg && Wc && bc, XB_ERR_ARG, "xb_augru: null tensor");
  XB_REQUIRE(batch >= 0 && T >= 0 && H >= 1, XB_ERR_ARG, "xb_augru: bad sizes");
  XB_REQUIRE(H <= 64, XB_ERR_LIMIT, "xb_augru: hidden size %d, at most 64 (weights are kept in shared memory)", H);
  XB_REQUIRE(dtype == XB_F32 || dtype == XB_F16, XB_ERR_UNSUPPORTED, "xb_augru: dtype %d", dtype);
  XB_REQUIRE(batch < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_augru: batch too large");
  if (batch == 0 || T == 0) return 0;
  const size_t smem = sizeof(float) * ((size_t)6 * H * H + 5 * H);
  static PerDeviceOnce attr;
  XB_SET_MAX_SMEM_ONCE(attr, 110 * 1024, (const void*)augru_kernel);
  const int threads = (2 * H + 31) / 32 * 32;
  launch_dependent(augru_kernel, (unsigned)batch, threads, smem, (cudaStream_t)s, x, att, y, T, H, Wg, bg, Wc, bc, dtype);
  return check_launch("augru_kernel");
}

extern "C" int xb_augru_shared(const void* x, const void* att, void* y_final, int32_t requests, int32_t n_cand, int32_t T,
                               int32_t H, const void* Wg, const void* bg, const void* Wc, const void* bc, int32_t engine,
                               xb_stream_t s) {
  XB_REQUIRE(x && att && y_final && Wg && bg && Wc && bc, XB_ERR_ARG, "xb_augru_shared: null tensor");
  XB_REQUIRE(requests >= 0 && n_cand >= 0 && T >= 1 && H >= 1, XB_ERR_ARG, "xb_augru_shared: bad sizes");
  XB_REQUIRE(H <= 64, XB_ERR_LIMIT, "xb_augru_shared: hidden size %d, at most 64", H);
  XB_REQUIRE(engine == XB_GEMM_AUTO || engine == XB_GEMM_SIMT || engine == XB_GEMM_TCGEN05, XB_ERR_ARG, "xb_augru_shared: engine %d", engine);
  if (requests == 0 || n_cand == 0) return 0;
  const bool tc = engine != XB_GEMM_SIMT && augru_tc_eligible(H, T);
  XB_REQUIRE(tc || engine != XB_GEMM_TCGEN05, XB_ERR_UNSUPPORTED,
             "xb_augru_shared: the tcgen05 engine takes an even H <= 64 whose padding to a multiple of 8 leaves 4 slots");
  AuParams p;
  memset(&p, 0, sizeof(p));
  p.x = (const __half*)x; p.att = (const __half*)att; p.y = (__half*)y_final;
  p.Wg = (const __half*)Wg; p.bg = (const __half*)bg; p.Wc = (const __half*)Wc; p.bc = (const __half*)bc;
  p.requests = requests; p.n_cand = n_cand; p.T = T; p.H = H;
  if (tc) return engine == XB_GEMM_AUTO && augru_mma_wanted(p) ? launch_augru_mma(p, (cudaStream_t)s) : launch_augru_tc(p, (cudaStream_t)s);
  XB_REQUIRE((int64_t)requests * n_cand < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_augru_shared: batch too large");
  switch ((H + 15) / 16) {
    case 1: return launch_augru_shared<1>(p, (cudaStream_t)s);
    case 2: return launch_augru_shared<2>(p, (cudaStream_t)s);
    case 3: return launch_augru_shared<3>(p, (cudaStream_t)s);
    default: return launch_augru_shared<4>(p, (cudaStream_t)s);
  }
}
