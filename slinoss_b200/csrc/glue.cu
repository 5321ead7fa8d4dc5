// Mixer glue around the scan in one pass each way: skip connection, (b,H,T,P) -> (b,T,H*P)
// re-layout and SiLU gate,
//     out[b,t,h*P+p] = (y[b,h,t,p] + skip[h*P+p] * u[b,h,t,p]) * silu(gate[b,t,h*P+p])
// (slinoss/layers/mixer.py:585-599 _apply_gate_skip, which runs five elementwise passes and a
// transposing copy), and its backward.  HBM-bound: 8 bytes per element forward (read y, u, gate,
// write out), 14 backward for half types.
//
// One thread owns 8 adjacent channels of one head (16 bytes of a half type) and walks a tile of
// tokens, several of them requested ahead; consecutive threads cover a (head, channel) row, so every access is a
// 128-byte segment.
// The backward accumulates d_skip per thread over its tile; a second kernel sums the per-tile
// partials in a fixed order (no atomics: results are bitwise repeatable).
#include <initializer_list>
#include <type_traits>

#include "common.cuh"

namespace slx {

constexpr int kGlueThreads = 256;
constexpr int kGlueAheadFwd = 4, kGlueAheadBwd = 2;  // tokens a thread requests before it uses the first

struct GlueDims {
  int batch, T, H, P;
  long long gate_stride;  // elements between tokens of gate (it may be a column slice of a wider row)
  long long gate_batch_stride;
  int skip_dtype;
  int tile, n_tiles;  // tokens per thread, tiles of the token axis
};

// A thread's share: 8 channels (16 bytes of a half type) of one tile of tokens.  Shares are numbered channels first
// and dealt to a flat grid, so that narrow layers fill their blocks.
struct GlueShare {
  int ch, b, tile_i, t0, t1;
  size_t yrow;  // element offset of (b, h, 0, p) in the head-major tensors
};
__device__ __forceinline__ bool glue_share(const GlueDims &d, GlueShare &s) {
  const unsigned C8 = (unsigned)(d.H * d.P) / 8;
  const unsigned idx = blockIdx.x * kGlueThreads + threadIdx.x;
  const unsigned r = idx / C8;
  s.ch = 8 * (int)(idx - r * C8);
  s.b = (int)(r / (unsigned)d.n_tiles);
  s.tile_i = (int)(r - (unsigned)s.b * d.n_tiles);
  if (s.b >= d.batch) return false;
  const int h = s.ch / d.P, p = s.ch - h * d.P;
  s.t0 = s.tile_i * d.tile;
  s.t1 = min(s.t0 + d.tile, d.T);
  s.yrow = (((size_t)s.b * d.H + h) * d.T) * d.P + p;
  return true;
}
// 1 / (1 + e^-x): half types take the fast reciprocal (error far below their rounding); with the full-precision
// division the two kernels were bound by instructions as much as by HBM.
template <typename T>
__device__ __forceinline__ float glue_sigmoid(float x) {
  if constexpr (sizeof(T) == 2) return __fdividef(1.f, 1.f + __expf(-x));
  else return 1.f / (1.f + __expf(-x));
}
// 8 values as they lie in memory
template <typename T>
struct alignas(16) Raw8 {
  T v[8];
};
template <typename T>
__device__ __forceinline__ Raw8<T> ldraw8(const T *p) {
  Raw8<T> r;
  *reinterpret_cast<uint4 *>(r.v) = *reinterpret_cast<const uint4 *>(p);
  if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4 *>(r.v + 4) = *reinterpret_cast<const uint4 *>(p + 4);
  return r;
}

template <typename T>
__device__ __forceinline__ void st8(T *p, const float (&v)[8]) {
  if constexpr (sizeof(T) == 2) {
    uint4 raw;
    T *e = reinterpret_cast<T *>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = from_f<T>(v[i]);
    *reinterpret_cast<uint4 *>(p) = raw;
  } else {
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// skip of 8 channels, rounded to the activation dtype (16-byte loads where its storage allows)
template <typename T>
__device__ __forceinline__ void load_skip(const void *skip, int dtype, int ch, float (&sk)[8]) {
  if (dtype != SLX_F32 && (reinterpret_cast<uintptr_t>(skip) & 15) == 0) {
    const Raw8<__half> r = ldraw8(static_cast<const __half *>(skip) + ch);  // bits of either half type
#pragma unroll
    for (int i = 0; i < 8; ++i) sk[i] = to_f(from_f<T>(load_as_f(r.v, dtype, i)));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) sk[i] = to_f(from_f<T>(load_as_f(skip, dtype, ch + i)));
  }
}

template <typename T>
__global__ void __launch_bounds__(kGlueThreads) gate_skip_fwd_kernel(const T *__restrict__ y, const T *__restrict__ u,
                                                            const T *__restrict__ gate, const void *__restrict__ skip,
                                                            T *__restrict__ out, GlueDims d) {
  constexpr int U = sizeof(T) == 2 ? kGlueAheadFwd : 2;
  GlueShare s;
  if (!glue_share(d, s)) return;
  float sk[8];
  load_skip<T>(skip, d.skip_dtype, s.ch, sk);
  const T *gb = gate + (size_t)s.b * d.gate_batch_stride + s.ch;
  T *ob = out + (size_t)s.b * d.T * d.H * d.P + s.ch;
  auto step = [&](auto n_tag, int t) {  // n tokens: all their loads, then the arithmetic
    constexpr int N = decltype(n_tag)::value;
    Raw8<T> yr[N], ur[N], gr[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      yr[k] = ldraw8(y + s.yrow + (size_t)(t + k) * d.P);
      ur[k] = ldraw8(u + s.yrow + (size_t)(t + k) * d.P);
      gr[k] = ldraw8(gb + (size_t)(t + k) * d.gate_stride);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        // the reference rounds skip*u, y + skip*u and silu(gate) to the activation dtype one after the other
        const float gv = to_f(gr[k].v[i]);
        const float a = to_f(from_f<T>(to_f(yr[k].v[i]) + to_f(from_f<T>(sk[i] * to_f(ur[k].v[i])))));
        const float sg = to_f(from_f<T>(gv * glue_sigmoid<T>(gv)));
        o[i] = a * sg;
      }
      st8<T>(ob + (size_t)(t + k) * d.H * d.P, o);
    }
  };
  int t = s.t0;
  for (; t + U <= s.t1; t += U) step(std::integral_constant<int, U>(), t);
  for (; t < s.t1; ++t) step(std::integral_constant<int, 1>(), t);
}

// d_out (b,T,H*P) -> dy, du (b,H,T,P), d_gate (b,T,H*P) contiguous, per-tile partials of d_skip
template <typename T>
__global__ void __launch_bounds__(kGlueThreads) gate_skip_bwd_kernel(const T *__restrict__ y, const T *__restrict__ u,
                                                            const T *__restrict__ gate, const void *__restrict__ skip,
                                                            const T *__restrict__ d_out, T *__restrict__ dy,
                                                            T *__restrict__ du, T *__restrict__ d_gate,
                                                            float *__restrict__ part, GlueDims d) {
  constexpr int U = sizeof(T) == 2 ? kGlueAheadBwd : 1;
  GlueShare s;
  if (!glue_share(d, s)) return;
  float sk[8], acc[8];
  load_skip<T>(skip, d.skip_dtype, s.ch, sk);
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  const T *gb = gate + (size_t)s.b * d.gate_batch_stride + s.ch;
  const size_t tb = (size_t)s.b * d.T * d.H * d.P + s.ch;
  auto step = [&](auto n_tag, int t) {
    constexpr int N = decltype(n_tag)::value;
    Raw8<T> yr[N], ur[N], gr[N], dr[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      yr[k] = ldraw8(y + s.yrow + (size_t)(t + k) * d.P);
      ur[k] = ldraw8(u + s.yrow + (size_t)(t + k) * d.P);
      gr[k] = ldraw8(gb + (size_t)(t + k) * d.gate_stride);
      dr[k] = ldraw8(d_out + tb + (size_t)(t + k) * d.H * d.P);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float o1[8], o2[8], o3[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float gv = to_f(gr[k].v[i]), go = to_f(dr[k].v[i]), uv = to_f(ur[k].v[i]);
        const float sig = glue_sigmoid<T>(gv);
        const float sg = to_f(from_f<T>(gv * sig));
        const float a = to_f(from_f<T>(to_f(yr[k].v[i]) + to_f(from_f<T>(sk[i] * uv))));
        const float g = go * sg;                          // gradient of y + skip*u
        o1[i] = g;
        o2[i] = g * sk[i];
        o3[i] = go * a * sig * (1.f + gv * (1.f - sig));  // d silu(g)/dg = sig (1 + g (1 - sig))
        acc[i] = fmaf(g, uv, acc[i]);
      }
      st8<T>(dy + s.yrow + (size_t)(t + k) * d.P, o1);
      st8<T>(du + s.yrow + (size_t)(t + k) * d.P, o2);
      st8<T>(d_gate + tb + (size_t)(t + k) * d.H * d.P, o3);
    }
  };
  int t = s.t0;
  for (; t + U <= s.t1; t += U) step(std::integral_constant<int, U>(), t);
  for (; t < s.t1; ++t) step(std::integral_constant<int, 1>(), t);
  float *pp = part + ((size_t)s.b * d.n_tiles + s.tile_i) * d.H * d.P + s.ch;
  reinterpret_cast<float4 *>(pp)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  reinterpret_cast<float4 *>(pp)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// d_skip[c] = sum over the partial rows, in a fixed order: 32 channels x 64 row groups per CTA, every thread adds
// the rows of its group (i = g, g + 64, ..., eight of them in flight), then the 64 group sums are added in order.
// (16 groups of one row at a time: 0.029 ms for 4096 rows of 1024 channels.)
__global__ void __launch_bounds__(512) gate_skip_reduce_kernel(const float *__restrict__ part, void *__restrict__ d_skip,
                                                               int skip_dtype, int n_part, int C) {
  constexpr int kGroups = 64, kAhead = 8;
  __shared__ float red[kGroups][33];
  const int cx = threadIdx.x & 7, g = threadIdx.x >> 3;
  const int c = blockIdx.x * 32 + 4 * cx;  // C is a multiple of 8
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](float4 v) {
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  };
  if (c < C) {
    const float *col = part + c;
    int i = g;
    for (; i + (kAhead - 1) * kGroups < n_part; i += kAhead * kGroups) {
      float4 v[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) v[k] = *reinterpret_cast<const float4 *>(col + (size_t)(i + k * kGroups) * C);
#pragma unroll
      for (int k = 0; k < kAhead; ++k) add(v[k]);
    }
    for (; i < n_part; i += kGroups) add(*reinterpret_cast<const float4 *>(col + (size_t)i * C));
  }
  red[g][4 * cx] = acc.x;
  red[g][4 * cx + 1] = acc.y;
  red[g][4 * cx + 2] = acc.z;
  red[g][4 * cx + 3] = acc.w;
  __syncthreads();
  // four groups of 16 per channel, then their four sums
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float tot = 0.f;
  if (w < 4) {
#pragma unroll
    for (int k = 0; k < 16; ++k) tot += red[16 * w + k][lane];
  }
  __syncthreads();
  if (w < 4) red[w][lane] = tot;
  __syncthreads();
  if (w == 0 && blockIdx.x * 32 + lane < C)
    store_as(d_skip, skip_dtype, blockIdx.x * 32 + lane, (red[0][lane] + red[1][lane]) + (red[2][lane] + red[3][lane]));
}

static int check_glue(const slx_glue_shape *s, GlueDims *d) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  SLX_REQUIRE(s->batch > 0 && s->T > 0 && s->heads > 0 && s->P > 0, SLX_E_SHAPE, "gate_skip: sizes must be positive");
  SLX_REQUIRE(s->P % 8 == 0, SLX_E_UNSUPPORTED, "gate_skip: head dim %d must be a multiple of 8", s->P);
  SLX_REQUIRE(s->dtype >= SLX_F32 && s->dtype <= SLX_F16, SLX_E_DTYPE, "gate_skip: bad dtype %d", s->dtype);
  SLX_REQUIRE(s->batch <= 65535, SLX_E_UNSUPPORTED, "gate_skip: batch exceeds 65535");
  SLX_REQUIRE(s->gate_stride >= (int64_t)s->heads * s->P && s->gate_stride % 8 == 0 && s->gate_batch_stride % 8 == 0,
              SLX_E_UNSUPPORTED, "gate_skip: gate strides must be multiples of 8 elements and cover a row");
  d->batch = s->batch; d->T = s->T; d->H = s->heads; d->P = s->P;
  d->gate_stride = s->gate_stride; d->gate_batch_stride = s->gate_batch_stride;
  return SLX_OK;
}

// Tokens a thread walks.  Forward: one step (4 tokens of a half type), so that short sequences fill the GPU and long
// ones have no thin last wave (32-token walks: 0.028 ms for b2 T1000 with 512 channels, 0.122 ms for b16 T4096 with
// 1024, the last third of it on half the SMs).  Backward: the walk also sums d_skip, one partial row per tile; it
// grows from 4 to 16 tokens (where the partials are 2 % of the traffic) while the threads of the call overfill the GPU.
static void glue_tile(GlueDims *d, bool bwd) {
  const long long C8 = (long long)d->H * d->P / 8, resident = (long long)kB200Sms * 1024;
  int tile = 4;
  while (bwd && tile < 16 && C8 * d->batch * ((d->T + tile - 1) / tile) > resident) tile *= 2;
  d->tile = tile;
  d->n_tiles = (d->T + tile - 1) / tile;
}
static unsigned glue_grid(const GlueDims &d) {
  const long long shares = (long long)d.H * d.P / 8 * d.n_tiles * d.batch;
  return (unsigned)((shares + kGlueThreads - 1) / kGlueThreads);
}

static bool glue_aligned(std::initializer_list<const void *> ptrs) {
  for (const void *p : ptrs)
    if (p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
  return true;
}

}  // namespace slx

using namespace slx;

#define SLX_GLUE_T(dt, ...)                                          \
  switch (dt) {                                                      \
    case SLX_F32: { using T_ = float; __VA_ARGS__; } break;          \
    case SLX_BF16: { using T_ = __nv_bfloat16; __VA_ARGS__; } break; \
    default: { using T_ = __half; __VA_ARGS__; } break;              \
  }

extern "C" {

int slx_gate_skip_fwd_as(const slx_glue_shape *s, const void *y, const void *u, const void *gate, const void *skip,
                         int32_t skip_dtype, void *out, void *stream) {
  GlueDims d;
  int rc = check_glue(s, &d);
  if (rc) return rc;
  SLX_REQUIRE(y && u && gate && skip && out, SLX_E_NULL, "gate_skip_fwd: NULL tensor");
  d.skip_dtype = skip_dtype;
  SLX_REQUIRE(glue_aligned({y, u, gate, out}), SLX_E_UNSUPPORTED, "gate_skip_fwd: pointers must be 16-byte aligned");
  glue_tile(&d, false);
  SLX_GLUE_T(s->dtype, {
    gate_skip_fwd_kernel<T_><<<glue_grid(d), kGlueThreads, 0, as_stream(stream)>>>((const T_ *)y, (const T_ *)u, (const T_ *)gate, skip,
                                                                 (T_ *)out, d);
  });
  return check_launch("gate_skip_fwd");
}
int slx_gate_skip_fwd(const slx_glue_shape *s, const void *y, const void *u, const void *gate, const float *skip,
                      void *out, void *stream) {
  return slx_gate_skip_fwd_as(s, y, u, gate, skip, SLX_F32, out, stream);
}

size_t slx_gate_skip_bwd_workspace_bytes(const slx_glue_shape *s) {
  GlueDims d;
  if (check_glue(s, &d)) return 0;
  glue_tile(&d, true);
  return sizeof(float) * (size_t)d.batch * d.n_tiles * d.H * d.P;
}

int slx_gate_skip_bwd_as(const slx_glue_shape *s, const void *y, const void *u, const void *gate, const void *skip,
                         int32_t skip_dtype, const void *d_out, void *dy, void *du, void *d_gate, void *d_skip,
                         void *workspace, size_t workspace_bytes, void *stream) {
  GlueDims d;
  int rc = check_glue(s, &d);
  if (rc) return rc;
  SLX_REQUIRE(y && u && gate && skip && d_out && dy && du && d_gate && d_skip, SLX_E_NULL, "gate_skip_bwd: NULL tensor");
  d.skip_dtype = skip_dtype;
  SLX_REQUIRE(glue_aligned({y, u, gate, d_out, dy, du, d_gate, workspace}), SLX_E_UNSUPPORTED,
              "gate_skip_bwd: pointers must be 16-byte aligned");
  const size_t need = slx_gate_skip_bwd_workspace_bytes(s);
  SLX_REQUIRE(workspace && workspace_bytes >= need, SLX_E_WORKSPACE, "gate_skip_bwd: workspace of %zu bytes needed",
              need);
  glue_tile(&d, true);
  float *part = static_cast<float *>(workspace);
  SLX_GLUE_T(s->dtype, {
    gate_skip_bwd_kernel<T_><<<glue_grid(d), kGlueThreads, 0, as_stream(stream)>>>((const T_ *)y, (const T_ *)u, (const T_ *)gate, skip,
                                                                 (const T_ *)d_out, (T_ *)dy, (T_ *)du, (T_ *)d_gate,
                                                                 part, d);
  });
  rc = check_launch("gate_skip_bwd");
  if (rc) return rc;
  const int C = d.H * d.P;
  gate_skip_reduce_kernel<<<(C + 31) / 32, 512, 0, as_stream(stream)>>>(part, d_skip, skip_dtype, d.batch * d.n_tiles,
                                                                         C);
  return check_launch("gate_skip_reduce");
}
int slx_gate_skip_bwd(const slx_glue_shape *s, const void *y, const void *u, const void *gate, const float *skip,
                      const void *d_out, void *dy, void *du, void *d_gate, float *d_skip, void *workspace,
                      size_t workspace_bytes, void *stream) {
  return slx_gate_skip_bwd_as(s, y, u, gate, skip, SLX_F32, d_out, dy, du, d_gate, d_skip, workspace, workspace_bytes,
                              stream);
}

}  // extern "C"
