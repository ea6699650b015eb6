// GRU and attention-gated GRU (AUGRU) over short behaviour sequences.
//
// One CTA owns one sequence and walks its T steps, so a sequence never leaves
// its SM and needs no inter-CTA synchronisation (the reference CUDA GRU spins on
// global atomics between blocks, blaze/blaze/operator/op/gru_op.cu:73-85; nothing
// here waits on another CTA). Latency-bound by design: throughput comes from
// batch-many independent CTAs.
#include <cstring>

#include "xb_common.cuh"
#include "xb_umma.cuh"

namespace xb {
namespace {

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

__device__ __forceinline__ float sigm(float v) { return 1.f / (1.f + expf(-v)); }

// x [B,T,H], y [B,T,H]; i2h, h2h [H,3H] (gate order r, z, candidate); biases [3H].
// Follows GRUKernel, blaze/blaze/operator/op/gru_op.cc:33-93: leading steps whose first H
// input pre-activations (before the bias) are all zero emit zeros and leave h at zero.
//
// What bounds it is the chain h(t) -> h(t+1); everything else is kept off that chain. The input products of up to
// GRU_CHUNK steps are made first, one gate column per thread with its weights in registers (they do not depend on h).
// Then a step is: four lanes per unit, each with a quarter of the unit's three recurrent columns in registers, read
// their part of h as 16-byte vectors, add up over the lanes with two shuffles, and all four evaluate the gates; the
// new h goes to the other of two buffers, so a step needs one barrier. 16 sequences of 100 steps, H = 36: 77 us,
// 156 before (weights in shared memory, three barriers a step).
constexpr int GRU_CHUNK = 64;
__host__ __device__ constexpr int gru_hp(int nv) { return 16 * nv; }          // h and x rows padded with zeros
template <typename T, int NV>
__global__ void __launch_bounds__(64 * NV) gru_kernel(const T* x, T* y, int steps, int H,
                                                      const T* __restrict__ i2h, const T* __restrict__ h2h,
                                                      const T* __restrict__ bi, const T* __restrict__ bh) {
  pdl_begin();
  constexpr int HP = gru_hp(NV);
  extern __shared__ __align__(16) float gru_sm[];
  float* xs = gru_sm;                              // [GRU_CHUNK][HP]
  float* pre = xs + GRU_CHUNK * HP;                // [GRU_CHUNK][3H]: input products with their bias
  __shared__ __align__(16) float hbuf[2][HP];
  __shared__ int nonzero[GRU_CHUNK];               // step has a non-zero among its first H input products
  const int tid = threadIdx.x, G = 3 * H;
  const int u = tid >> 2, l = tid & 3;             // recurrence: unit and quarter
  const bool unit = u < H;
  const int64_t b = blockIdx.x;
  float wi[HP];                                    // column tid of i2h
  float wh[3][4 * NV];                             // rows 4 * (4 i + l) .. + 3 of the unit's columns
#pragma unroll
  for (int k = 0; k < HP; ++k) wi[k] = (k < H && tid < G) ? to_f32<T>(i2h[k * G + tid]) : 0.f;
#pragma unroll
  for (int g = 0; g < 3; ++g)
#pragma unroll
    for (int i = 0; i < 4 * NV; ++i) {
      const int k = 4 * (4 * (i >> 2) + l) + (i & 3);
      wh[g][i] = (unit && k < H) ? to_f32<T>(h2h[k * G + g * H + u]) : 0.f;
    }
  const float bij = tid < G ? to_f32<T>(bi[tid]) : 0.f;
  float bhu[3];
#pragma unroll
  for (int g = 0; g < 3; ++g) bhu[g] = unit ? to_f32<T>(bh[g * H + u]) : 0.f;
  for (int i = tid; i < 2 * HP; i += blockDim.x) (&hbuf[0][0])[i] = 0.f;
  bool started = false;
  float h = 0.f;
  for (int t0 = 0; t0 < steps; t0 += GRU_CHUNK) {
    const int n = min(GRU_CHUNK, steps - t0);
    __syncthreads();                               // the last chunk's rows have been used
    const T* xb = x + (b * steps + t0) * H;
    for (int i = tid; i < n * HP; i += blockDim.x) {
      const int t = i / HP, k = i - t * HP;
      xs[i] = k < H ? to_f32<T>(xb[t * H + k]) : 0.f;
    }
    for (int i = tid; i < n; i += blockDim.x) nonzero[i] = 0;
    __syncthreads();
    if (tid < G) {
#pragma unroll 4
      for (int t = 0; t < n; ++t) {
        float p = 0.f;
#pragma unroll
        for (int k = 0; k < HP; k += 4) {
          const float4 v = *reinterpret_cast<const float4*>(xs + t * HP + k);
          p = fmaf(v.x, wi[k], p); p = fmaf(v.y, wi[k + 1], p); p = fmaf(v.z, wi[k + 2], p); p = fmaf(v.w, wi[k + 3], p);
        }
        if (tid < H && p != 0.f) nonzero[t] = 1;
        pre[t * G + tid] = p + bij;
      }
    }
    __syncthreads();
    for (int t = 0; t < n; ++t) {
      const int64_t at = (b * steps + t0 + t) * H + u;
      if (!started) started = nonzero[t] != 0;     // the same for every thread
      if (!started) {
        if (unit && l == 0) y[at] = from_f32<T>(0.f);
        continue;
      }
      float pr = 0.f, pz = 0.f, pc = 0.f;
      if (unit) { pr = pre[t * G + u]; pz = pre[t * G + H + u]; pc = pre[t * G + 2 * H + u]; }
      const float4* hv = reinterpret_cast<const float4*>(hbuf[t & 1]);
      float a[3][2] = {};
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float4 v = hv[4 * i + l];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          a[g][0] = fmaf(v.x, wh[g][4 * i], a[g][0]);
          a[g][1] = fmaf(v.y, wh[g][4 * i + 1], a[g][1]);
          a[g][0] = fmaf(v.z, wh[g][4 * i + 2], a[g][0]);
          a[g][1] = fmaf(v.w, wh[g][4 * i + 3], a[g][1]);
        }
      }
      float s[3];
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        s[g] = a[g][0] + a[g][1];
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], 1);
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], 2);
        s[g] += bhu[g];
      }
      const float r = sigm(pr + s[0]);
      const float z = sigm(pz + s[1]);
      const float c = tanhf(pc + r * s[2]);
      h = c + z * (h - c);
      if (unit && l == 0) {
        hbuf[(t + 1) & 1][u] = h;
        y[at] = from_f32<T>(h);
      }
      __syncthreads();
    }
    // an odd number of steps leaves h in the second buffer: the next chunk counts its steps from zero again, and every
    // chunk but the last has GRU_CHUNK (even) steps, so it starts in the first
  }
}

// AUGRU after VecAttGRUCell.call (xdl-algorithm-solution/DIEN/script/utils.py:139-207):
// [r|u] = sigmoid([x,h] Wg + bg); c = tanh([x, r*h] Wc + bc); u' = (1 - a_t) u; h' = u' h + (1 - u') c.
// Wg [2H, 2H] (rows x then h; columns r then u), Wc [2H, H]; att [B, T].
// `share` > 0: the input sequence is shared by groups of `share` consecutive batch entries (x is [B / share, T, H],
// the candidates of one request), and only the final state is written (y is [B, H]).
__global__ void augru_kernel(const void* x, const void* att, void* y, int T, int H, const void* Wg_, const void* bg_,
                             const void* Wc_, const void* bc_, int dt, int share) {
  pdl_begin();
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
    const int64_t xbase = share > 0 ? ((b / share) * T + t) * H : base;
    if (j < H) xs[j] = load_as_f32(x, xbase + j, dt);
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
      if (share <= 0) store_from_f32(y, base + j, dt, out);
      else if (t == T - 1) store_from_f32(y, b * H + j, dt, out);
    }
    __syncthreads();
    if (j < H) h[j] = out;
  }
}

template <typename T, int NV>
int launch_gru_nv(const T* x, T* y, int64_t batch, int steps, int H, const T* i2h, const T* h2h, const T* bi, const T* bh,
                  cudaStream_t s) {
  const size_t smem = sizeof(float) * GRU_CHUNK * (size_t)(gru_hp(NV) + 3 * H);
  static PerDeviceOnce attr;                       // per instantiation
  XB_SET_MAX_SMEM_ONCE(attr, sizeof(float) * GRU_CHUNK * 4 * gru_hp(NV), (const void*)gru_kernel<T, NV>);
  launch_dependent(gru_kernel<T, NV>, (unsigned)batch, (4 * H + 31) / 32 * 32, smem, s, x, y, steps, H, i2h, h2h, bi, bh);
  return check_launch("gru_kernel");
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

#include "xb_augru_tc.cuh"

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
  XB_REQUIRE(H <= 64, XB_ERR_LIMIT, "xb_gru: hidden size %d, at most 64 (weights are kept in shared memory)", H);
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
  launch_dependent(augru_kernel, (unsigned)batch, threads, smem, (cudaStream_t)s, x, att, y, T, H, Wg, bg, Wc, bc, dtype, 0);
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
  if (tc) {
    AuParams p;
    memset(&p, 0, sizeof(p));
    p.x = (const __half*)x; p.att = (const __half*)att; p.y = (__half*)y_final;
    p.Wg = (const __half*)Wg; p.bg = (const __half*)bg; p.Wc = (const __half*)Wc; p.bc = (const __half*)bc;
    p.requests = requests; p.n_cand = n_cand; p.T = T; p.H = H;
    return launch_augru_tc(p, (cudaStream_t)s);
  }
  const int64_t batch = (int64_t)requests * n_cand;
  XB_REQUIRE(batch < ((int64_t)1 << 31), XB_ERR_LIMIT, "xb_augru_shared: batch too large");
  const size_t smem = sizeof(float) * ((size_t)6 * H * H + 5 * H);
  static PerDeviceOnce attr;
  XB_SET_MAX_SMEM_ONCE(attr, 110 * 1024, (const void*)augru_kernel);
  const int threads = (2 * H + 31) / 32 * 32;
  launch_dependent(augru_kernel, (unsigned)batch, threads, smem, (cudaStream_t)s, x, att, y_final, T, H, Wg, bg, Wc, bc, XB_F16, n_cand);
  return check_launch("augru_kernel");
}
