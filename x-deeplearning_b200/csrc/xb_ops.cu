// Stand-alone activation, normalisation, elementwise and data-movement
// operators for graphs whose ops were not fused into a GEMM epilogue, plus the
// library's error/version plumbing. All are HBM-bound streaming kernels:
// grid-stride loops sized to a multiple of the SM count.
#include <cstring>

#include "xb_common.cuh"

namespace xb {

static thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}
void clear_error() { g_err[0] = 0; }

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

static inline unsigned stream_grid(int64_t work_items, int per_block) {
  int64_t blocks = (work_items + per_block - 1) / per_block;
  int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (unsigned)blocks;
}

__global__ void dice_kernel(const void* x, void* y, int64_t size, int c, const void* gamma,
                            const void* mean, const void* var, int nosqrt, int dt) {
  pdl_begin();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x) {
    int col = (int)(i % c);
    float v = load_as_f32(x, i, dt);
    float r = act_dice(v, load_as_f32(gamma, col, dt), load_as_f32(mean, col, dt),
                       dice_rstd(load_as_f32(var, col, dt), nosqrt));
    store_from_f32(y, i, dt, r);
  }
}

__global__ void prelu_kernel(const void* x, void* y, int64_t size, const void* w, int64_t inner, int dt, int wdt) {
  pdl_begin();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x)
    store_from_f32(y, i, dt, act_prelu(load_as_f32(x, i, dt), load_as_f32(w, i % inner, wdt)));
}

__global__ void sigmoid_kernel(const void* x, void* y, int64_t size, int dt) {
  pdl_begin();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x)
    store_from_f32(y, i, dt, act_sigmoid(load_as_f32(x, i, dt)));
}

__global__ void batchnorm_kernel(const void* x, void* y, int64_t size, int c, const void* gamma, const void* beta,
                                 const void* mean, const void* var, float eps, int nosqrt, int dt) {
  pdl_begin();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x) {
    int col = (int)(i % c);
    float vr = load_as_f32(var, col, dt);
    float xn = (load_as_f32(x, i, dt) - load_as_f32(mean, col, dt)) / (nosqrt ? vr : sqrtf(vr + eps));
    store_from_f32(y, i, dt, load_as_f32(gamma, col, dt) * xn + load_as_f32(beta, col, dt));
  }
}

// one thread per (outer, inner) pair walks the c axis three times (max, sum, divide)
__global__ void softmax_kernel(const void* x, void* y, int64_t n, int c, int64_t w, int dt) {
  pdl_begin();
  const int64_t total = n * w;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t base = (i / w) * c * w + (i % w);
    float m = load_as_f32(x, base, dt);
    for (int j = 1; j < c; ++j) m = fmaxf(m, load_as_f32(x, base + (int64_t)j * w, dt));
    float s = 0.f;
    for (int j = 0; j < c; ++j) s += __expf(load_as_f32(x, base + (int64_t)j * w, dt) - m);
    for (int j = 0; j < c; ++j)
      store_from_f32(y, base + (int64_t)j * w, dt, __expf(load_as_f32(x, base + (int64_t)j * w, dt) - m) / s);
  }
}

// Contiguous rows (w == 1) of 16 and more columns: one warp per row, so that a row is read in coalesced pieces, and up to
// 256 columns stay in registers between the three passes. 16 000 rows of 100 fp32: 7.3 us, 34 before (one thread per row
// touches 32 rows with every load).
template <int PER>
__global__ void __launch_bounds__(256) softmax_rows_kernel(const void* x, void* y, __half* y16, int64_t n, int c, int dt) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * 8;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < n; r += warps) {
    const int64_t base = r * c;
    float v[PER], m = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = lane + 32 * i;
      v[i] = j < c ? load_as_f32(x, base + j, dt) : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) m = fmaxf(m, v[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = lane + 32 * i < c ? __expf(v[i] - m) : 0.f;
      s += v[i];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = lane + 32 * i;
      if (j >= c) continue;
      v[i] /= s;
      store_from_f32(y, base + j, dt, v[i]);
      if (y16) y16[base + j] = __float2half_rn(v[i]);
    }
  }
}

// The same for fp32 rows of whole, aligned 16-byte pieces, eight lanes a row and four columns a lane at a time: a quarter of the
// shuffles. Many rows of up to 128 columns alone: with few rows the two are the same, with more columns or single loads a lane's
// chain is longer than a warp's (33 523 rows of 137 24 us, 19 a warp a row). 16 000 rows of 100 4.5 us, 6.4 a warp a row; 74 000 11.1,
// 24.6; 2048 2.4 either way.
template <int PER4>
__global__ void __launch_bounds__(256) softmax_f32_kernel(const float* x, float* y, __half* y16, int64_t n, int c) {
  pdl_begin();
  const bool y16_vec = (reinterpret_cast<uintptr_t>(y16) & 7) == 0;
  const int l = threadIdx.x & 7, sub = threadIdx.x >> 3 & 3;
  const int64_t rows = (int64_t)gridDim.x * 32;
  for (int64_t at = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 5) * 4; at < n; at += rows) {       // the same for a warp: its shuffles stay whole
    const int64_t r = at + sub;
    const bool in = r < n;
    const float* xr = x + r * c;
    float v[PER4][4], m = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER4; ++i) {
      const int j = 4 * (l + 8 * i);
      const float4 q = in && j < c ? *reinterpret_cast<const float4*>(xr + j) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      v[i][0] = q.x; v[i][1] = q.y; v[i][2] = q.z; v[i][3] = q.w;
    }
#pragma unroll
    for (int i = 0; i < PER4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) m = fmaxf(m, v[i][e]);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[i][e] = 4 * (l + 8 * i) + e < c ? __expf(v[i][e] - m) : 0.f;
        s += v[i][e];
      }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (!in) continue;
#pragma unroll
    for (int i = 0; i < PER4; ++i) {
      const int j = 4 * (l + 8 * i);
      if (j >= c) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[i][e] /= s;
      *reinterpret_cast<float4*>(y + r * c + j) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
      if (!y16) continue;
      const __half2 lo = __floats2half2_rn(v[i][0], v[i][1]), hi = __floats2half2_rn(v[i][2], v[i][3]);
      if (y16_vec) {
        *reinterpret_cast<uint2*>(y16 + r * c + j) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      } else {
        y16[r * c + j] = __low2half(lo); y16[r * c + j + 1] = __high2half(lo);
        y16[r * c + j + 2] = __low2half(hi); y16[r * c + j + 3] = __high2half(hi);
      }
    }
  }
}

// Rows of 16 to 256 columns. y16, where given, receives the fp16 rounding of an fp32 y, which saves the pass that would convert it
// (16 000 rows of 100: 4.7 us, 9.5 as two launches).
static int launch_softmax_rows(const void* x, void* y, __half* y16, int64_t n, int c, int dt, cudaStream_t s) {
  if (dt == XB_F32 && c % 4 == 0 && c <= 128 && n >= 2048 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
    const float* xf = static_cast<const float*>(x);
    float* yf = static_cast<float*>(y);
    if (c <= 64) launch_dependent(softmax_f32_kernel<2>, stream_grid(n, 32), 256, 0, s, xf, yf, y16, n, c);
    else launch_dependent(softmax_f32_kernel<4>, stream_grid(n, 32), 256, 0, s, xf, yf, y16, n, c);
    return check_launch("softmax_f32_kernel");
  }
  const unsigned grid = stream_grid(n, 8);
  if (c <= 64) launch_dependent(softmax_rows_kernel<2>, grid, 256, 0, s, x, y, y16, n, c, dt);
  else if (c <= 128) launch_dependent(softmax_rows_kernel<4>, grid, 256, 0, s, x, y, y16, n, c, dt);
  else launch_dependent(softmax_rows_kernel<8>, grid, 256, 0, s, x, y, y16, n, c, dt);
  return check_launch("softmax_rows_kernel");
}

struct EwParams {
  int op, dt;
  const void *a, *b, *c;
  void* y;
  int64_t as[4], bs[4], cs[4], shape[4];
};

__device__ __forceinline__ float ew_apply(int op, float av, float bv) {
  switch (op) {
    case XB_EW_ADD: return av + bv;
    case XB_EW_SUB: return av - bv;
    case XB_EW_MUL: return av * bv;
    case XB_EW_DIV: return av / bv;
    case XB_EW_MAX: return fmaxf(av, bv);
    case XB_EW_MIN: return fminf(av, bv);
    case XB_EW_EQ: return av == bv ? 1.f : 0.f;
    default: return av != bv ? 1.f : 0.f;
  }
}

__global__ void elementwise_kernel(const __grid_constant__ EwParams p) {
  pdl_begin();
  const int64_t total = p.shape[0] * p.shape[1] * p.shape[2] * p.shape[3];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i;
    const int64_t i3 = r % p.shape[3]; r /= p.shape[3];
    const int64_t i2 = r % p.shape[2]; r /= p.shape[2];
    const int64_t i1 = r % p.shape[1]; r /= p.shape[1];
    const int64_t i0 = r;
    const int64_t ia = i0 * p.as[0] + i1 * p.as[1] + i2 * p.as[2] + i3 * p.as[3];
    const int64_t ib = i0 * p.bs[0] + i1 * p.bs[1] + i2 * p.bs[2] + i3 * p.bs[3];
    float out;
    if (p.op == XB_EW_WHERE) {
      const int64_t ic = i0 * p.cs[0] + i1 * p.cs[1] + i2 * p.cs[2] + i3 * p.cs[3];
      const int32_t cond = reinterpret_cast<const int32_t*>(p.a)[ia];
      out = cond ? load_as_f32(p.b, ib, p.dt) : load_as_f32(p.c, ic, p.dt);
    } else if (p.op == XB_EW_BROADCAST_TO) {
      out = load_as_f32(p.a, ia, p.dt);
    } else {
      out = ew_apply(p.op, load_as_f32(p.a, ia, p.dt), load_as_f32(p.b, ib, p.dt));
    }
    store_from_f32(p.y, i, p.dt, out);
  }
}

// Four fp32 elements of the innermost axis per thread: 16-byte accesses (an operand that repeats along that axis is read
// once), 32-bit index arithmetic and one decomposition of the index per four elements; the kernel above spends its time
// on four 64-bit divisions per element. The launcher merges axes that every operand walks contiguously and sees to
// alignment. [500, 100, 36] - [1, 100, 36]: 3.3 us, 14 before
__global__ void __launch_bounds__(256) elementwise4_kernel(const __grid_constant__ EwParams p) {
  pdl_begin();
  const uint32_t s1 = (uint32_t)p.shape[1], s2 = (uint32_t)p.shape[2], s3 = (uint32_t)p.shape[3] / 4;
  const uint32_t total = (uint32_t)p.shape[0] * s1 * s2 * s3;
  const bool rep_a = p.as[3] == 0, rep_b = p.bs[3] == 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    uint32_t r = i / s3;
    const uint32_t i3 = i - r * s3;
    uint32_t q = r / s2;
    const uint32_t i2 = r - q * s2;
    const uint32_t i0 = q / s1, i1 = q - i0 * s1;
    auto load4 = [&](const void* base, const int64_t* st, bool rep) {
      const float* f = reinterpret_cast<const float*>(base) + (int64_t)i0 * st[0] + (int64_t)i1 * st[1] + (int64_t)i2 * st[2];
      if (rep) { const float v = *f; return make_float4(v, v, v, v); }
      return *reinterpret_cast<const float4*>(f + 4 * i3);
    };
    const float4 a = load4(p.a, p.as, rep_a);
    float4 o = a;
    if (p.op != XB_EW_BROADCAST_TO) {
      const float4 b = load4(p.b, p.bs, rep_b);
      o = make_float4(ew_apply(p.op, a.x, b.x), ew_apply(p.op, a.y, b.y), ew_apply(p.op, a.z, b.z), ew_apply(p.op, a.w, b.w));
    }
    reinterpret_cast<float4*>(p.y)[i] = o;
  }
}

__global__ void copy2d_kernel(const void* src, int64_t src_ld, int sdt, void* dst, int64_t dst_ld, int ddt,
                              int64_t rows, int64_t cols) {
  pdl_begin();
  const int64_t total = rows * cols;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    // 32-bit division where it will do: the 64-bit one is most of the instructions of an element
    const int64_t r = total < ((int64_t)1 << 31) ? (int64_t)((uint32_t)i / (uint32_t)cols) : i / cols, c = i - r * cols;
    if (sdt == XB_I32 && ddt == XB_I32)
      reinterpret_cast<int32_t*>(dst)[r * dst_ld + c] = reinterpret_cast<const int32_t*>(src)[r * src_ld + c];
    else if (sdt == XB_I64 && ddt == XB_I64)
      reinterpret_cast<int64_t*>(dst)[r * dst_ld + c] = reinterpret_cast<const int64_t*>(src)[r * src_ld + c];
    else
      store_from_f32(dst, r * dst_ld + c, ddt, load_as_f32(src, r * src_ld + c, sdt));
  }
}

// Same-type copies of rows whose pieces of sizeof(V) bytes are aligned in source and destination: one piece per thread and
// 32-bit index arithmetic (element by element the kernel above is bound by its 64-bit division). 50 000 rows of 36 fp32
// into rows of 144: 1.9 us, 5 before
template <typename V>
__global__ void __launch_bounds__(256) copy2d_vec_kernel(const V* src, int64_t src_ld, V* dst, int64_t dst_ld, uint32_t total, uint32_t cols) {
  pdl_begin();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t r = i / cols, c = i - r * cols;
    dst[(int64_t)r * dst_ld + c] = src[(int64_t)r * src_ld + c];
  }
}

// fp32 <-> fp16 copies, four elements per thread (16 bytes on one side, 8 on the other)
template <bool TO_HALF>
__global__ void __launch_bounds__(256) copy2d_convert_kernel(const void* src, int64_t src_ld, void* dst, int64_t dst_ld, uint32_t total, uint32_t cols) {
  pdl_begin();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t r = i / cols, c = i - r * cols;
    if (TO_HALF) {
      const float4 v = reinterpret_cast<const float4*>(src)[(int64_t)r * src_ld + c];
      const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
      reinterpret_cast<uint2*>(dst)[(int64_t)r * dst_ld + c] =
          make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    } else {
      const uint2 v = reinterpret_cast<const uint2*>(src)[(int64_t)r * src_ld + c];
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
      reinterpret_cast<float4*>(dst)[(int64_t)r * dst_ld + c] = make_float4(a.x, a.y, b.x, b.y);
    }
  }
}

__global__ void reduce_sum_kernel(const void* x, void* y, int64_t outer, int64_t r, int64_t inner, int dt) {
  pdl_begin();
  const int64_t total = outer * inner;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t o = i / inner, in = i - o * inner;
    float s = 0.f;
    // eight loads in flight, added in order
    int64_t j = 0;
    for (; j + 8 <= r; j += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = load_as_f32(x, (o * r + j + u) * inner + in, dt);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; j < r; ++j) s += load_as_f32(x, (o * r + j) * inner + in, dt);
    store_from_f32(y, i, dt, s);
  }
}

// W [K,N] row-major (ld ldw) -> out [N, ldk] with zero padding of k in [K, ldk)
__global__ void pack_kmajor_kernel(const void* W, int wdt, int K, int N, int64_t ldw, void* out, int odt,
                                   int64_t ldk, int64_t stride_w, int64_t stride_out) {
  const int64_t b = blockIdx.y;
  const int64_t total = (int64_t)N * ldk;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i / ldk, k = i - n * ldk;
    float v = k < K ? load_as_f32(W, b * stride_w + k * ldw + n, wdt) : 0.f;
    store_from_f32(out, b * stride_out + i, odt, v);
  }
}

// one CTA per (request, 64-candidate slab); his_sum is rebuilt per CTA from the T k rows. The row is
// produced two columns (one 32-bit store) at a time when d and du are even; every feature segment then
// starts on a 4-byte boundary in X and in q / att.
__global__ void __launch_bounds__(256) din_tower_input_kernel(const __half* user, int64_t ldu, const __half* q,
                                                              int64_t ldq, const __half* k, int64_t ldk,
                                                              const __half* att, int64_t ldatt, __half* X, int64_t ldx,
                                                              int n_cand, int T, int d, int du, int pairs_ok) {
  pdl_begin();
  extern __shared__ float hs[];      // [d] his_sum, then [du] user row
  float* us = hs + d;
  const int r = blockIdx.y;
  // his_sum: the block's threads split the T steps (groups of d threads take every G-th step), partial
  // sums meet in shared memory and are added in group order, so the result does not depend on timing
  float* part = us + du;             // [G][d]
  const int G = max(1, min((int)blockDim.x / d, 8));
  if ((int)threadIdx.x < G * d) {
    const int gi = threadIdx.x / d, e = threadIdx.x - gi * d;
    float s = 0.f;
    // eight steps requested together, added in order
    for (int t = gi; t < T; t += 8 * G) {
      __half v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = t + u * G < T ? k[((int64_t)r * T + t + u * G) * ldk + e] : __float2half(0.f);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t + u * G < T) s += __half2float(v[u]);
    }
    part[gi * d + e] = s;
  }
  for (int e = threadIdx.x; e < du; e += blockDim.x) us[e] = __half2float(user[(int64_t)r * ldu + e]);
  __syncthreads();
  for (int e = threadIdx.x; e < d; e += blockDim.x) {
    float s = 0.f;
    for (int gi = 0; gi < G; ++gi) s += part[gi * d + e];
    hs[e] = s;
  }
  __syncthreads();
  const int n0 = blockIdx.x * 64;
  const int rows = min(64, n_cand - n0);
  if (pairs_ok == 2) {
    // Four columns (8 bytes) at a time. A thread keeps its columns and takes every few rows, so the columns' place and
    // what is the same for all rows are worked out once. 16 000 rows of 328 columns: 16 us
    // behind the AUGRU, 19 without asking for rows ahead
    const int wq = (int)(ldx >> 2), step = max(1, (int)blockDim.x / wq);
    for (int q0 = threadIdx.x; q0 < step * wq; q0 += blockDim.x) {
      const int r0 = q0 / wq, c = (q0 - r0 * wq) * 4;
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      int seg = -1, e = 0;                             // -1: the same four values in every row
      if (c < du) {
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = us[c + u];
      } else if (c < du + 5 * d) {
        seg = (c - du) / d;
        e = (c - du) - seg * d;
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = hs[e + u];
        if (seg == 1) seg = -1;
      }
      const __half* src = seg == 3 ? att + e : q + e;
      const int64_t ld = seg == 3 ? ldatt : ldq, row0 = (int64_t)r * n_cand + n0;
      constexpr int U = 8;                             // rows requested together (a store would hold back the loads behind it)
      for (int nl0 = r0; nl0 < rows; nl0 += U * step) {
        uint2 raw[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int nl = nl0 + k * step;
          raw[k] = make_uint2(0u, 0u);
          if (seg >= 0 && nl < rows) raw[k] = *reinterpret_cast<const uint2*>(src + (row0 + nl) * ld);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int nl = nl0 + k * step;
          if (nl >= rows) continue;
          float v[4] = {f[0], f[1], f[2], f[3]};
          if (seg >= 0) {
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw[k].x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw[k].y));
            const float x[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = seg == 2 ? x[u] * f[u] : seg == 4 ? x[u] - f[u] : x[u];
          }
          const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
          uint2 w;
          w.x = *reinterpret_cast<const uint32_t*>(&a); w.y = *reinterpret_cast<const uint32_t*>(&b);
          *reinterpret_cast<uint2*>(X + (row0 + nl) * ldx + c) = w;
        }
      }
    }
    return;
  }
  if (pairs_ok) {
    const int wp = (int)(ldx >> 1);                    // half2 units per row
    for (int idx = threadIdx.x; idx < rows * wp; idx += blockDim.x) {
      const int n = n0 + idx / wp, c = (idx % wp) * 2;
      const int64_t row = (int64_t)r * n_cand + n;
      float2 v = make_float2(0.f, 0.f);
      if (c < du) v = make_float2(us[c], us[c + 1]);
      else if (c < du + 5 * d) {
        const int seg = (c - du) / d, e = (c - du) - seg * d;
        if (seg == 1) v = make_float2(hs[e], hs[e + 1]);
        else if (seg == 3) v = __half22float2(*reinterpret_cast<const __half2*>(att + row * ldatt + e));
        else {
          const float2 qv = __half22float2(*reinterpret_cast<const __half2*>(q + row * ldq + e));
          if (seg == 0) v = qv;
          else if (seg == 2) v = make_float2(qv.x * hs[e], qv.y * hs[e + 1]);
          else v = make_float2(qv.x - hs[e], qv.y - hs[e + 1]);
        }
      }
      *reinterpret_cast<__half2*>(X + row * ldx + c) = __floats2half2_rn(v.x, v.y);
    }
    return;
  }
  const int width = (int)ldx;
  for (int idx = threadIdx.x; idx < rows * width; idx += blockDim.x) {
    const int n = n0 + idx / width, c = idx % width;
    const int64_t row = (int64_t)r * n_cand + n;
    float v = 0.f;
    if (c < du) v = us[c];
    else if (c < du + 5 * d) {
      const int seg = (c - du) / d, e = (c - du) % d;
      const float qv = __half2float(q[row * ldq + e]);
      if (seg == 0) v = qv;
      else if (seg == 1) v = hs[e];
      else if (seg == 2) v = qv * hs[e];
      else if (seg == 3) v = __half2float(att[row * ldatt + e]);
      else v = qv - hs[e];
    }
    X[row * ldx + c] = __float2half_rn(v);
  }
}

// Split form: per-request columns [user | his_sum] once per request, per-candidate columns
// [q | q*his_sum | att | q-his_sum] per candidate. Same CTA shape as above.
__global__ void __launch_bounds__(256) din_tower_split_kernel(const __half* user, int64_t ldu, const __half* q,
                                                              int64_t ldq, const __half* k, int64_t ldk,
                                                              const __half* att, int64_t ldatt, __half* Xu, int64_t ldxu,
                                                              __half* Xc, int64_t ldxc, int n_cand, int T, int d, int du,
                                                              int pairs_ok) {
  pdl_begin();
  extern __shared__ float hs[];      // [d] his_sum, then [G][d] partial sums
  float* part = hs + d;
  const int r = blockIdx.y;
  const int G = max(1, min((int)blockDim.x / d, 8));
  if ((int)threadIdx.x < G * d) {
    const int gi = threadIdx.x / d, e = threadIdx.x - gi * d;
    float s = 0.f;
    // eight steps requested together, added in order
    for (int t = gi; t < T; t += 8 * G) {
      __half v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = t + u * G < T ? k[((int64_t)r * T + t + u * G) * ldk + e] : __float2half(0.f);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t + u * G < T) s += __half2float(v[u]);
    }
    part[gi * d + e] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < d; e += blockDim.x) {
    float s = 0.f;
    for (int gi = 0; gi < G; ++gi) s += part[gi * d + e];
    hs[e] = s;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int c = threadIdx.x; c < (int)ldxu; c += blockDim.x) {
      __half v = __float2half(0.f);
      if (c < du) v = user[(int64_t)r * ldu + c];
      else if (c < du + d) v = __float2half_rn(hs[c - du]);
      Xu[(int64_t)r * ldxu + c] = v;
    }
  }
  const int n0 = blockIdx.x * 64;
  const int rows = min(64, n_cand - n0);
  if (pairs_ok) {
    const int wp = (int)(ldxc >> 1);                   // half2 units per row
    for (int idx = threadIdx.x; idx < rows * wp; idx += blockDim.x) {
      const int n = n0 + idx / wp, c = (idx % wp) * 2;
      const int64_t row = (int64_t)r * n_cand + n;
      float2 v = make_float2(0.f, 0.f);
      if (c < 4 * d) {
        const int seg = c / d, e = c - seg * d;
        if (seg == 2) v = __half22float2(*reinterpret_cast<const __half2*>(att + row * ldatt + e));
        else {
          const float2 qv = __half22float2(*reinterpret_cast<const __half2*>(q + row * ldq + e));
          if (seg == 0) v = qv;
          else if (seg == 1) v = make_float2(qv.x * hs[e], qv.y * hs[e + 1]);
          else v = make_float2(qv.x - hs[e], qv.y - hs[e + 1]);
        }
      }
      *reinterpret_cast<__half2*>(Xc + row * ldxc + c) = __floats2half2_rn(v.x, v.y);
    }
    return;
  }
  const int width = (int)ldxc;
  for (int idx = threadIdx.x; idx < rows * width; idx += blockDim.x) {
    const int n = n0 + idx / width, c = idx % width;
    const int64_t row = (int64_t)r * n_cand + n;
    float v = 0.f;
    if (c < 4 * d) {
      const int seg = c / d, e = c % d;
      if (seg == 2) v = __half2float(att[row * ldatt + e]);
      else {
        const float qv = __half2float(q[row * ldq + e]);
        v = seg == 0 ? qv : (seg == 1 ? qv * hs[e] : qv - hs[e]);
      }
    }
    Xc[row * ldxc + c] = __float2half_rn(v);
  }
}

static bool float_dtype(int dt) { return dt == XB_F32 || dt == XB_F16 || dt == XB_BF16; }

}  // namespace xb

using namespace xb;

extern "C" const char* xb_last_error(void) { return g_err; }
extern "C" const char* xb_version(void) { return "xdlb200 0.1 (sm_100a)"; }

extern "C" int xb_dice(const void* x, void* y, int64_t rows, int32_t c, const void* gamma, const void* mean,
                       const void* var, int32_t nosqrt, int32_t dtype, xb_stream_t s) {
  XB_REQUIRE(x && y && gamma && mean && var && c > 0 && rows >= 0, XB_ERR_ARG, "xb_dice: bad arguments");
  XB_REQUIRE(float_dtype(dtype), XB_ERR_UNSUPPORTED, "xb_dice: dtype %d", dtype);
  if (rows == 0) return 0;
  launch_dependent(dice_kernel, stream_grid(rows * c, 256), 256, 0, (cudaStream_t)s, x, y, rows * c, c, gamma, mean, var, nosqrt, dtype);
  return check_launch("dice_kernel");
}

extern "C" int xb_prelu(const void* x, void* y, int64_t size, const void* w, int64_t inner, int32_t dtype,
                        int32_t w_dtype, xb_stream_t s) {
  XB_REQUIRE(x && y && w && inner > 0 && size >= 0, XB_ERR_ARG, "xb_prelu: bad arguments");
  XB_REQUIRE(float_dtype(dtype) && float_dtype(w_dtype), XB_ERR_UNSUPPORTED, "xb_prelu: dtype %d/%d", dtype, w_dtype);
  if (size == 0) return 0;
  launch_dependent(prelu_kernel, stream_grid(size, 256), 256, 0, (cudaStream_t)s, x, y, size, w, inner, dtype, w_dtype);
  return check_launch("prelu_kernel");
}

extern "C" int xb_sigmoid(const void* x, void* y, int64_t size, int32_t dtype, xb_stream_t s) {
  XB_REQUIRE(x && y && size >= 0, XB_ERR_ARG, "xb_sigmoid: bad arguments");
  XB_REQUIRE(float_dtype(dtype), XB_ERR_UNSUPPORTED, "xb_sigmoid: dtype %d", dtype);
  if (size == 0) return 0;
  launch_dependent(sigmoid_kernel, stream_grid(size, 256), 256, 0, (cudaStream_t)s, x, y, size, dtype);
  return check_launch("sigmoid_kernel");
}

extern "C" int xb_softmax(const void* x, void* y, int64_t n, int32_t c, int64_t w, int32_t dtype, xb_stream_t s) {
  XB_REQUIRE(x && y && n >= 0 && c > 0 && w > 0, XB_ERR_ARG, "xb_softmax: bad arguments");
  XB_REQUIRE(float_dtype(dtype), XB_ERR_UNSUPPORTED, "xb_softmax: dtype %d", dtype);
  if (n == 0) return 0;
  if (w == 1 && c >= 16 && c <= 256) return launch_softmax_rows(x, y, nullptr, n, c, dtype, (cudaStream_t)s);
  launch_dependent(softmax_kernel, stream_grid(n * w, 128), 128, 0, (cudaStream_t)s, x, y, n, c, w, dtype);
  return check_launch("softmax_kernel");
}

extern "C" int xb_softmax_scores(const float* x, float* y, void* y16, int64_t n, int32_t c, xb_stream_t s) {
  XB_REQUIRE(x && y && y16 && n >= 0 && c > 0, XB_ERR_ARG, "xb_softmax_scores: bad arguments");
  if (n == 0) return 0;
  if (c >= 16 && c <= 256) return launch_softmax_rows(x, y, (__half*)y16, n, c, XB_F32, (cudaStream_t)s);
  if (int rc = xb_softmax(x, y, n, c, 1, XB_F32, s)) return rc;
  return xb_copy2d(y, c, XB_F32, y16, c, XB_F16, n, c, s);
}

extern "C" int xb_batchnorm(const void* x, void* y, int64_t size, int32_t c, const void* gamma, const void* beta,
                            const void* mean, const void* var, float eps, int32_t nosqrt, int32_t dtype,
                            xb_stream_t s) {
  XB_REQUIRE(x && y && gamma && beta && mean && var && c > 0 && size >= 0, XB_ERR_ARG, "xb_batchnorm: bad arguments");
  XB_REQUIRE(float_dtype(dtype), XB_ERR_UNSUPPORTED, "xb_batchnorm: dtype %d", dtype);
  if (size == 0) return 0;
  launch_dependent(batchnorm_kernel, stream_grid(size, 256), 256, 0, (cudaStream_t)s, x, y, size, c, gamma, beta, mean, var, eps, nosqrt, dtype);
  return check_launch("batchnorm_kernel");
}

extern "C" int xb_elementwise(int32_t op, const void* a, const int64_t* as, const void* b, const int64_t* bs,
                              const void* c, const int64_t* cs, void* y, const int64_t* shape, int32_t dtype,
                              xb_stream_t s) {
  XB_REQUIRE(op >= XB_EW_ADD && op <= XB_EW_WHERE, XB_ERR_UNSUPPORTED, "xb_elementwise: op %d", op);
  XB_REQUIRE(a && as && y && shape, XB_ERR_ARG, "xb_elementwise: null pointer");
  XB_REQUIRE(op == XB_EW_BROADCAST_TO || (b && bs), XB_ERR_ARG, "xb_elementwise: second operand missing");
  XB_REQUIRE(op != XB_EW_WHERE || (c && cs), XB_ERR_ARG, "xb_elementwise: third operand missing");
  XB_REQUIRE(float_dtype(dtype) || dtype == XB_I32, XB_ERR_UNSUPPORTED, "xb_elementwise: dtype %d", dtype);
  EwParams p;
  memset(&p, 0, sizeof(p));
  p.op = op; p.dt = dtype; p.a = a; p.b = b; p.c = c; p.y = y;
  int64_t total = 1;
  for (int i = 0; i < 4; ++i) {
    XB_REQUIRE(shape[i] >= 0, XB_ERR_ARG, "xb_elementwise: negative extent");
    p.shape[i] = shape[i]; p.as[i] = as[i];
    p.bs[i] = bs ? bs[i] : 0; p.cs[i] = cs ? cs[i] : 0;
    total *= shape[i];
  }
  if (total == 0) return 0;
  if (dtype == XB_F32 && op != XB_EW_WHERE && total < ((int64_t)1 << 31)) {
    // merge an axis into the one inside it where both operands step over it as over one axis (the output is dense)
    EwParams m = p;
    const bool two = op != XB_EW_BROADCAST_TO;
    for (int i = 2; i >= 0; --i) {
      const bool merge = m.shape[i] == 1 || (m.as[i] == m.as[3] * m.shape[3] && (!two || m.bs[i] == m.bs[3] * m.shape[3]));
      if (!merge) break;
      m.shape[3] *= m.shape[i];
      for (int j = i; j > 0; --j) { m.shape[j] = m.shape[j - 1]; m.as[j] = m.as[j - 1]; m.bs[j] = m.bs[j - 1]; }
      m.shape[0] = 1; m.as[0] = m.bs[0] = 0;
      ++i;                                            // the next outer axis is at the same place now
      if (m.shape[0] * m.shape[1] * m.shape[2] == 1) break;
    }
    auto fits = [&](const void* base, const int64_t* st) {
      if (st[3] == 0) return true;
      return st[3] == 1 && (reinterpret_cast<uintptr_t>(base) & 15) == 0 && st[0] % 4 == 0 && st[1] % 4 == 0 && st[2] % 4 == 0;
    };
    if (m.shape[3] % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0 && fits(a, m.as) && (!two || fits(b, m.bs))) {
      launch_dependent(elementwise4_kernel, stream_grid(total / 4, 256), 256, 0, (cudaStream_t)s, m);
      return check_launch("elementwise4_kernel");
    }
  }
  launch_dependent(elementwise_kernel, stream_grid(total, 256), 256, 0, (cudaStream_t)s, p);
  return check_launch("elementwise_kernel");
}

extern "C" int xb_copy2d(const void* src, int64_t src_ld, int32_t sdt, void* dst, int64_t dst_ld, int32_t ddt,
                         int64_t rows, int64_t cols, xb_stream_t s) {
  XB_REQUIRE(src && dst && rows >= 0 && cols >= 0, XB_ERR_ARG, "xb_copy2d: bad arguments");
  XB_REQUIRE(dtype_size(sdt) && dtype_size(ddt), XB_ERR_UNSUPPORTED, "xb_copy2d: dtype %d -> %d", sdt, ddt);
  XB_REQUIRE((sdt == XB_I64) == (ddt == XB_I64), XB_ERR_UNSUPPORTED, "xb_copy2d: int64 converts to nothing else");
  if (rows * cols == 0) return 0;
  if (sdt == ddt) {
    // widest piece that divides the row and both pitches and to which both ends are aligned
    const int64_t es = (int64_t)dtype_size(sdt);
    const uintptr_t bits = (uintptr_t)src | (uintptr_t)dst | (uintptr_t)(src_ld * es) | (uintptr_t)(dst_ld * es) | (uintptr_t)(cols * es);
    const int64_t w = bits % 16 == 0 ? 16 : bits % 8 == 0 ? 8 : bits % 4 == 0 ? 4 : 2;
    const int64_t pieces = rows * cols * es / w;
    if (bits % 2 == 0 && pieces < ((int64_t)1 << 30)) {
      const unsigned grid = stream_grid(pieces, 256);
      const uint32_t pc = (uint32_t)(cols * es / w);
      const int64_t sl = src_ld * es / w, dl = dst_ld * es / w;
      const cudaStream_t st = (cudaStream_t)s;
      if (w == 16) launch_dependent(copy2d_vec_kernel<uint4>, grid, 256, 0, st, (const uint4*)src, sl, (uint4*)dst, dl, (uint32_t)pieces, pc);
      else if (w == 8) launch_dependent(copy2d_vec_kernel<uint2>, grid, 256, 0, st, (const uint2*)src, sl, (uint2*)dst, dl, (uint32_t)pieces, pc);
      else if (w == 4) launch_dependent(copy2d_vec_kernel<uint32_t>, grid, 256, 0, st, (const uint32_t*)src, sl, (uint32_t*)dst, dl, (uint32_t)pieces, pc);
      else launch_dependent(copy2d_vec_kernel<uint16_t>, grid, 256, 0, st, (const uint16_t*)src, sl, (uint16_t*)dst, dl, (uint32_t)pieces, pc);
      return check_launch("copy2d_vec_kernel");
    }
  }
  const bool to_half = sdt == XB_F32 && ddt == XB_F16;
  if ((to_half || (sdt == XB_F16 && ddt == XB_F32)) && src_ld % 4 == 0 && dst_ld % 4 == 0 && cols % 4 == 0 &&
      ((uintptr_t)src & (to_half ? 15 : 7)) == 0 && ((uintptr_t)dst & (to_half ? 7 : 15)) == 0 && rows * cols < ((int64_t)1 << 31)) {
    const uint32_t n = (uint32_t)(rows * cols / 4);
    launch_dependent(to_half ? copy2d_convert_kernel<true> : copy2d_convert_kernel<false>, stream_grid(n, 256), 256, 0, (cudaStream_t)s,
                     src, src_ld / 4, dst, dst_ld / 4, n, (uint32_t)(cols / 4));
    return check_launch("copy2d_convert_kernel");
  }
  launch_dependent(copy2d_kernel, stream_grid(rows * cols, 256), 256, 0, (cudaStream_t)s, src, src_ld, sdt, dst, dst_ld, ddt, rows, cols);
  return check_launch("copy2d_kernel");
}

// One CTA column per descriptor, blockIdx.y walks the copy in 32 KB pieces; 16-byte vectors when both ends
// and the length allow it, single bytes otherwise (id lists and segment counts of odd lengths).
constexpr int64_t COPY_PIECE = 32 * 1024;
__global__ void copy_segments_kernel(const xb_copy_item* __restrict__ items) {
  pdl_begin();
  const xb_copy_item it = items[blockIdx.x];
  const int64_t begin = (int64_t)blockIdx.y * COPY_PIECE;
  if (begin >= it.bytes) return;
  const int64_t n = min(COPY_PIECE, it.bytes - begin);
  const uint8_t* src = reinterpret_cast<const uint8_t*>(it.src) + begin;
  uint8_t* dst = reinterpret_cast<uint8_t*>(it.dst) + begin;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
    const int64_t nv = n / 16;
    for (int64_t i = threadIdx.x; i < nv; i += blockDim.x)
      reinterpret_cast<uint4*>(dst)[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
    for (int64_t i = nv * 16 + threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  } else {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  }
}

extern "C" int xb_copy_segments(const xb_copy_item* items, int32_t n_items, int64_t max_bytes, xb_stream_t s) {
  XB_REQUIRE(n_items >= 0 && max_bytes >= 0 && (n_items == 0 || items), XB_ERR_ARG, "xb_copy_segments: bad arguments");
  if (n_items == 0 || max_bytes == 0) return 0;
  const int64_t pieces = (max_bytes + COPY_PIECE - 1) / COPY_PIECE;
  XB_REQUIRE(pieces <= 65535, XB_ERR_LIMIT, "xb_copy_segments: a copy of %lld bytes is too long for one call", (long long)max_bytes);
  dim3 grid((unsigned)n_items, (unsigned)pieces);
  launch_dependent(copy_segments_kernel, grid, 256, 0, (cudaStream_t)s, items);
  return check_launch("copy_segments_kernel");
}

extern "C" int xb_reduce_sum(const void* x, void* y, int64_t outer, int64_t r, int64_t inner, int32_t dtype,
                             xb_stream_t s) {
  XB_REQUIRE(x && y && outer >= 0 && r >= 0 && inner >= 0, XB_ERR_ARG, "xb_reduce_sum: bad arguments");
  XB_REQUIRE(float_dtype(dtype), XB_ERR_UNSUPPORTED, "xb_reduce_sum: dtype %d", dtype);
  if (outer * inner == 0) return 0;
  launch_dependent(reduce_sum_kernel, stream_grid(outer * inner, 128), 128, 0, (cudaStream_t)s, x, y, outer, r, inner, dtype);
  return check_launch("reduce_sum_kernel");
}

extern "C" int xb_pack_weight_kmajor(const void* W, int32_t w_dtype, int32_t K, int32_t N, int64_t ldw, void* out,
                                     int32_t out_dtype, int64_t ldk, int32_t batch, int64_t stride_w,
                                     int64_t stride_out, xb_stream_t s) {
  XB_REQUIRE(W && out && K > 0 && N > 0 && batch > 0, XB_ERR_ARG, "xb_pack_weight_kmajor: bad arguments");
  XB_REQUIRE(ldk >= K && ldw >= N, XB_ERR_ARG, "xb_pack_weight_kmajor: leading dimensions too small");
  XB_REQUIRE(float_dtype(w_dtype) && float_dtype(out_dtype), XB_ERR_UNSUPPORTED, "xb_pack_weight_kmajor: dtype");
  XB_REQUIRE(batch <= 65535, XB_ERR_LIMIT, "xb_pack_weight_kmajor: batch %d", batch);
  dim3 grid(stream_grid((int64_t)N * ldk, 256), batch);
  pack_kmajor_kernel<<<grid, 256, 0, (cudaStream_t)s>>>(W, w_dtype, K, N, ldw, out, out_dtype, ldk, stride_w, stride_out);
  return check_launch("pack_kmajor_kernel");
}

extern "C" int xb_din_tower_input(const void* user, int64_t ldu, const void* q, int64_t ldq, const void* k,
                                  int64_t ldk, const void* att, int64_t ldatt, void* X, int64_t ldx,
                                  int32_t requests, int32_t n_cand, int32_t T, int32_t d, int32_t du,
                                  xb_stream_t s) {
  XB_REQUIRE(user && q && k && att && X, XB_ERR_ARG, "xb_din_tower_input: null tensor");
  XB_REQUIRE(requests >= 0 && n_cand >= 0 && T >= 0 && d > 0 && du >= 0, XB_ERR_ARG, "xb_din_tower_input: bad sizes");
  XB_REQUIRE(d <= 256 && du <= 4096, XB_ERR_LIMIT, "xb_din_tower_input: d <= 256 and du <= 4096");
  XB_REQUIRE(ldx >= du + 5 * d && ldu >= du && ldq >= d && ldk >= d && ldatt >= d, XB_ERR_ARG,
             "xb_din_tower_input: leading dimension too small");
  XB_REQUIRE(requests <= 65535 && ldx <= 65536, XB_ERR_LIMIT, "xb_din_tower_input: more than 65535 requests per call");
  if (requests == 0 || n_cand == 0) return 0;
  dim3 grid((n_cand + 63) / 64, requests);
  // 32-bit accesses need even segment widths and leading dimensions and 4-byte aligned bases
  const int pairs_ok = d % 2 == 0 && du % 2 == 0 && ldx % 2 == 0 && ldq % 2 == 0 && ldatt % 2 == 0 &&
                       (((uintptr_t)q | (uintptr_t)att | (uintptr_t)X) & 3) == 0;
  // 64-bit ones need the same of multiples of four
  const int quads_ok = d % 4 == 0 && du % 4 == 0 && ldx % 4 == 0 && ldq % 4 == 0 && ldatt % 4 == 0 &&
                       (((uintptr_t)q | (uintptr_t)att | (uintptr_t)X) & 7) == 0;
  launch_dependent(din_tower_input_kernel, grid, 256, sizeof(float) * (9 * d + du + 2), (cudaStream_t)s, 
      (const __half*)user, ldu, (const __half*)q, ldq, (const __half*)k, ldk, (const __half*)att, ldatt, (__half*)X,
      ldx, n_cand, T, d, du, quads_ok ? 2 : pairs_ok);
  return check_launch("din_tower_input_kernel");
}

extern "C" int xb_din_tower_input_split(const void* user, int64_t ldu, const void* q, int64_t ldq, const void* k,
                                        int64_t ldk, const void* att, int64_t ldatt, void* Xu, int64_t ldxu, void* Xc,
                                        int64_t ldxc, int32_t requests, int32_t n_cand, int32_t T, int32_t d, int32_t du,
                                        xb_stream_t s) {
  XB_REQUIRE(user && q && k && att && Xu && Xc, XB_ERR_ARG, "xb_din_tower_input_split: null tensor");
  XB_REQUIRE(requests >= 0 && n_cand >= 0 && T >= 0 && d > 0 && du >= 0, XB_ERR_ARG, "xb_din_tower_input_split: bad sizes");
  XB_REQUIRE(d <= 256 && du <= 4096, XB_ERR_LIMIT, "xb_din_tower_input_split: d <= 256 and du <= 4096");
  XB_REQUIRE(ldxu >= du + d && ldxc >= 4 * d && ldu >= du && ldq >= d && ldk >= d && ldatt >= d, XB_ERR_ARG,
             "xb_din_tower_input_split: leading dimension too small");
  XB_REQUIRE(requests <= 65535 && ldxc <= 65536 && ldxu <= 65536, XB_ERR_LIMIT,
             "xb_din_tower_input_split: more than 65535 requests per call");
  if (requests == 0) return 0;
  dim3 grid(n_cand > 0 ? (n_cand + 63) / 64 : 1, requests);
  const int pairs_ok = d % 2 == 0 && ldxc % 2 == 0 && ldq % 2 == 0 && ldatt % 2 == 0 &&
                       (((uintptr_t)q | (uintptr_t)att | (uintptr_t)Xc) & 3) == 0;
  launch_dependent(din_tower_split_kernel, grid, 256, sizeof(float) * (9 * d + 2), (cudaStream_t)s, 
      (const __half*)user, ldu, (const __half*)q, ldq, (const __half*)k, ldk, (const __half*)att, ldatt, (__half*)Xu,
      ldxu, (__half*)Xc, ldxc, n_cand, T, d, du, pairs_ok);
  return check_launch("din_tower_split_kernel");
}
