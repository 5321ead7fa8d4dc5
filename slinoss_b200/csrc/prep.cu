// SLinOSSScanPrep forward/backward for sm_100a: bandwidth-bound, one lane group
// per (batch, head, token) row, 128-bit vector loads/stores, deterministic
// two-level reductions for the parameter gradients.
//
// Forward map (slinoss/layers/scanprep.py:351-357):
//   U  = value.view(b,T,H,P).permute(0,2,1,3)
//   B,C = interleave(rms_norm(bc) * scale)       (scanprep.py:297-336)
//   M,K = coefficient map of the 13-wide params row (scanprep.py:208-286,
//         ops/scanprep/reference.py:26-57)
#include <initializer_list>

#include "common.cuh"
#include "prep_coef.cuh"

namespace slx {

// VJP of coef_forward: dp[13] from (dM, dKprev, dKcurr)
__device__ __forceinline__ void coef_backward(const CoefCtx &c, const PrepHyper &h, float2 dm, float2 dkp, float2 dkc,
                                              float *dp) {
  const float d_dt = h.dt_max - h.dt_min, d_r = h.r_max - h.r_min;
  auto rdot = [](float2 a, float2 g) { return a.x * g.x + a.y * g.y; };
  float2 dkps = cscale(dkp, c.mix_kp), dkpl = cscale(dkp, 1.f - c.mix_kp);
  float dmix_kp = rdot(csub(c.kps, c.kpl), dkp);
  float2 dkcs = cscale(dkc, c.mix_kc), dkcl = cscale(dkc, 1.f - c.mix_kc);
  float dmix_kc = rdot(csub(c.kcs, c.kcl), dkc);
  float2 dk2 = cscale(csub(dkps, dkcs), c.dt);
  float2 dk1 = cscale(dkcs, c.dt);
  float ddt = rdot(c.k2, dkps) + rdot(csub(c.k1, c.k2), dkcs);
  float2 k1p, k2p;
  const float2 z = c.z;
  k1p = c.k2;  // d/dz (e^z-1)/z = kappa2, in both branches
  if (c.small) k2p = c.k2p;                                      // series (prep_coef.cuh)
  else k2p = cdiv(csub(c.rho, cscale(c.k2, 2.f)), z);            // d/dz (e^z(z-1)+1)/z^2 = (e^z - 2 kappa2)/z
  // dz = conj(k1') dk1 + conj(k2') dk2 + conj(rho) dM
  float2 dz = cadd(cadd(cmul(cconj(k1p), dk1), cmul(cconj(k2p), dk2)), cmul(cconj(c.rho), dm));
  float dr = dz.x / c.r;
  float dtheta = dz.y;
  float dth_d = (1.f - c.mix_th) * dtheta, dth_s = c.mix_th * dtheta;
  float dmix_th = (c.th_struct - c.th_direct) * dtheta;
  float dr_d = (1.f - c.mix_r) * dr, dr_s = c.mix_r * dr;
  float dmix_r = (c.r_struct - c.r_direct) * dr;
  float dgamma = dr_s * d_r * c.e_gdt * (-c.dt);
  ddt += dr_s * d_r * c.e_gdt * (-c.gamma);
  float domega = dth_s * c.dt;
  ddt += dth_s * c.omega;
  auto dsig = [](float s) { return s * (1.f - s); };
  dp[0] = ddt * d_dt * dsig(c.dt_u);
  dp[1] = dgamma * c.sig_p1;
  dp[2] = domega;
  dp[3] = dr_d * d_r * dsig(c.r_dir_u);
  dp[4] = dth_d * h.theta_bound * (1.f - c.th_t * c.th_t);
  dp[5] = dmix_r * dsig(c.mix_r);
  dp[6] = dmix_th * dsig(c.mix_th);
  dp[7] = dmix_kp * dsig(c.mix_kp);
  dp[8] = dmix_kc * dsig(c.mix_kc);
  dp[9] = h.k_max * (1.f - c.tk[0] * c.tk[0]) * dkpl.x;
  dp[10] = h.k_max * (1.f - c.tk[1] * c.tk[1]) * dkpl.y;
  dp[11] = h.k_max * (1.f - c.tk[2] * c.tk[2]) * dkcl.x;
  dp[12] = h.k_max * (1.f - c.tk[3] * c.tk[3]) * dkcl.y;
}

// ---- vector access ------------------------------------------------------------
template <typename T, int VEC>
__device__ __forceinline__ void load_vec(const T *p, float (&v)[VEC]) {
  if constexpr (VEC * sizeof(T) == 32 && sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else if constexpr (VEC * sizeof(T) == 16) {
    uint4 raw = *reinterpret_cast<const uint4 *>(p);
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = to_f(e[i]);
  } else if constexpr (VEC * sizeof(T) == 8) {
    uint2 raw = *reinterpret_cast<const uint2 *>(p);
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = to_f(e[i]);
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = to_f(p[i]);
  }
}
template <typename T, int VEC>
__device__ __forceinline__ void store_vec(T *p, const float (&v)[VEC]) {
  if constexpr (VEC * sizeof(T) == 16) {
    uint4 raw;
    T *e = reinterpret_cast<T *>(&raw);
#pragma unroll
    for (int i = 0; i < VEC; ++i) e[i] = from_f<T>(v[i]);
    *reinterpret_cast<uint4 *>(p) = raw;
  } else if constexpr (VEC * sizeof(T) == 8) {
    uint2 raw;
    T *e = reinterpret_cast<T *>(&raw);
#pragma unroll
    for (int i = 0; i < VEC; ++i) e[i] = from_f<T>(v[i]);
    *reinterpret_cast<uint2 *>(p) = raw;
  } else if constexpr (VEC * sizeof(T) == 32 && sizeof(T) == 4) {
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i) p[i] = from_f<T>(v[i]);
  }
}

// VEC adjacent RMS-norm scales of plane j, head h
template <int VEC>
__device__ __forceinline__ void load_scale(const PrepParams &pp, int h, int j, int N, int n0, float (&v)[VEC]) {
  const void *base = scale_plane(pp, j);
  const size_t e = scale_index(pp, h, j, N, n0);
  if (pp.dtype == SLX_BF16) load_vec<__nv_bfloat16, VEC>(static_cast<const __nv_bfloat16 *>(base) + e, v);
  else if (pp.dtype == SLX_F16) load_vec<__half, VEC>(static_cast<const __half *>(base) + e, v);
  else load_vec<float, VEC>(static_cast<const float *>(base) + e, v);
}

// ---- the 13-value parameter row of one (batch, head, token) ---------------------------------
// Half types: the row is 26 bytes at an arbitrary 2-byte offset.  `wide` loads the two or three
// aligned 16-byte vectors that cover it and picks the 13 values out by the (per-thread) offset;
// the caller passes wide = true only when every such vector lies inside the tensor (base and row
// stride multiples of 16 bytes, row width a multiple of 16 bytes).  Stores pair the values into
// 4-byte words wherever the address allows: 7 stores instead of 13.
template <typename T, int O>
__device__ __forceinline__ void pick13(const uint32_t (&w)[12], float (&p)[13]) {
#pragma unroll
  for (int i = 0; i < 13; ++i) {
    const uint32_t word = w[(O + i) >> 1];
    const unsigned short hbits = ((O + i) & 1) ? (unsigned short)(word >> 16) : (unsigned short)(word & 0xffffu);
    T v;
    *reinterpret_cast<unsigned short *>(&v) = hbits;
    p[i] = to_f(v);
  }
}
template <typename T>
__device__ __forceinline__ void load_row13(const T *pr, bool wide, float (&p)[13]) {
  if constexpr (sizeof(T) == 2) {
    if (wide) {
      const uintptr_t a = reinterpret_cast<uintptr_t>(pr);
      const uint4 *base = reinterpret_cast<const uint4 *>(a & ~uintptr_t(15));
      const int o = (int)((a & 15) >> 1);
      const uint4 v0 = base[0], v1 = base[1];
      uint4 v2 = make_uint4(0, 0, 0, 0);
      if (o > 3) v2 = base[2];  // elements o .. o+12 reach past the second vector
      const uint32_t w[12] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w};
      switch (o) {
        case 0: pick13<T, 0>(w, p); break;
        case 1: pick13<T, 1>(w, p); break;
        case 2: pick13<T, 2>(w, p); break;
        case 3: pick13<T, 3>(w, p); break;
        case 4: pick13<T, 4>(w, p); break;
        case 5: pick13<T, 5>(w, p); break;
        case 6: pick13<T, 6>(w, p); break;
        default: pick13<T, 7>(w, p); break;
      }
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < 13; ++i) p[i] = to_f(pr[i]);
}
template <typename T>
__device__ __forceinline__ void store_row13(T *pr, const float (&v)[13]) {
  if constexpr (sizeof(T) == 2) {
    auto pair = [&](int i) {
      T lo = from_f<T>(v[i]), hi = from_f<T>(v[i + 1]);
      const uint32_t word = (uint32_t)(*reinterpret_cast<unsigned short *>(&lo)) |
                            ((uint32_t)(*reinterpret_cast<unsigned short *>(&hi)) << 16);
      *reinterpret_cast<uint32_t *>(pr + i) = word;
    };
    if ((reinterpret_cast<uintptr_t>(pr) & 3) == 0) {
#pragma unroll
      for (int i = 0; i < 12; i += 2) pair(i);
      pr[12] = from_f<T>(v[12]);
    } else {
      pr[0] = from_f<T>(v[0]);
#pragma unroll
      for (int i = 1; i < 13; i += 2) pair(i);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 13; ++i) pr[i] = from_f<T>(v[i]);
  }
}

template <int G>
__device__ __forceinline__ float group_sum_f(float v) {
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

struct PrepDims {
  int batch, T, H, P, N;
  int normalize;
  long long vs, ps, bs;  // row strides (elements)
  int wide_params;        // params rows start on 16-byte boundaries (half types)
};
// the 16-byte vectors that cover head h's 13 values lie inside its row of the tensor
__device__ __forceinline__ bool row13_wide(const PrepDims &d, int h) {
  return d.wide_params && (26 * (h + 1) + 15) / 16 * 16 <= 26 * d.H;
}

// ---- asynchronous copies of one lane's 16-byte slice (AL = alignment of the source: 16, or 8 as two halves) ----
template <int AL>
__device__ __forceinline__ void copy_slice(void *smem_dst, const void *gsrc) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  if constexpr (AL == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gsrc) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(gsrc) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8), "l"((const char *)gsrc + 8) : "memory");
  }
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Sums over the G lanes of a group of four values at once: the lanes first trade values until each holds one of the
// four partial sums (3 shuffles; even lanes values 0 and 1, odd lanes 2 and 3), finish that one (log2 G - 2), apply `f` to it and hand the result round (4).
template <int G, typename F>
__device__ __forceinline__ void group_sum4(float (&v)[4], F f) {
  static_assert(G >= 4, "four lanes hold the four sums");
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2;
  const float p0 = (b0 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[2], 1);
  const float p1 = (b0 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, b0 ? v[1] : v[3], 1);
  float w = (b1 ? p1 : p0) + __shfl_xor_sync(0xffffffffu, b1 ? p0 : p1, 2);
#pragma unroll
  for (int off = 4; off < G; off <<= 1) w += __shfl_xor_sync(0xffffffffu, w, off);
  w = f(w);
  const int base = lane & ~3;
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __shfl_sync(0xffffffffu, w, base + (j >> 1) + ((j & 1) << 1));
}

// Forward, rows that one 16-byte slice per lane covers (VEC elements per lane, G lanes per row, G * VEC >= N and P).
// HBM-bound.  Rows are ordered (b, h, t), so that a CTA's consecutive rows write contiguous output.
//   * Every lane copies its own five slices of a row (value and the four bc planes) into a ring of kPrepRing rows,
//     so that two rows per group are on their way while one is worked on, without registers held for them and
//     without a barrier; the first two are requested before the coefficient map, whose ~500 scalar instructions
//     (one row per thread) run while they travel.
//   * Rows per CTA shrink from 256 to 32 while the CTAs do not fill the GPU: a short prompt is latency-bound.
//   * The RMS scales of the group's head stay in registers until the head changes.
// b16 T4096 16 heads N128: 0.406 ms (0.94 of the copy rate; 0.504 with rows requested one ahead through registers, 16
// lanes per row whatever its width and 256 rows per CTA); b2 T1000 8 heads N64: 0.009 ms (0.025).
constexpr int kPrepRing = 3;
template <typename T, int VEC, int G, int AL>
__global__ void __launch_bounds__(256, 3) scanprep_fwd_kernel(const T *__restrict__ value, const T *__restrict__ params,
                                                              const T *__restrict__ bc, PrepParams pp,
                                                              T *__restrict__ U, float *__restrict__ M,
                                                              float *__restrict__ K, T *__restrict__ Bo,
                                                              T *__restrict__ Co, PrepDims d, PrepHyper hp,
                                                              int rows_per_cta) {
  constexpr int NG = 256 / G;  // row groups per CTA
  extern __shared__ uint4 prep_ring[];  // [kPrepRing][5][256 threads]
  __shared__ float sbias[258 * 7];      // biases of the CTA's (batch, head)s: at most 257, two for T >= 256
  const int q = threadIdx.x % G, grp = threadIdx.x / G;
  const int n0 = q * VEC;
  const int D = 2 * d.N;
  const long long n_rows = (long long)d.batch * d.H * d.T;
  const long long row0 = (long long)blockIdx.x * rows_per_cta;
  const int rows = (int)min((long long)rows_per_cta, n_rows - row0);
  const int bh0 = (int)(row0 / d.T), tfirst = (int)(row0 - (long long)bh0 * d.T);
  const bool on_n = n0 < d.N, on_p = n0 < d.P;

  // the group's walk: rows grp, grp + NG, ... of the CTA
  struct Walk {
    int t, bh;
    long long in_row;
    int h;
  };
  auto settle = [&](Walk &w) {
    while (w.t >= d.T) {
      w.t -= d.T;
      ++w.bh;
    }
    const int b = w.bh / d.H;
    w.h = w.bh - b * d.H;
    w.in_row = (long long)b * d.T + w.t;
  };
  auto advance = [&](Walk &w) {
    w.t += NG;
    if (w.t < d.T) w.in_row += NG;
    else settle(w);
  };
  Walk ahead{tfirst + grp, bh0, 0, 0};
  settle(ahead);
  uint4 *slot = prep_ring + threadIdx.x;
  auto request = [&](int i) {  // row grp + i * NG into ring slot i % kPrepRing
    if (grp + i * NG < rows) {
      uint4 *s = slot + (i % kPrepRing) * 5 * 256;
      if (on_n) {
        const T *bcr = bc + ahead.in_row * d.bs + (long long)ahead.h * 4 * d.N + n0;
#pragma unroll
        for (int j = 0; j < 4; ++j) copy_slice<AL>(s + j * 256, bcr + j * d.N);
      }
      if (on_p) copy_slice<AL>(s + 4 * 256, value + ahead.in_row * d.vs + (long long)ahead.h * d.P + n0);
      advance(ahead);
    }
    copy_commit();
  };
#pragma unroll
  for (int i = 0; i < kPrepRing - 1; ++i) request(i);

  // ---- coefficient map, one row per thread ----
  {
    const int n_bh = (tfirst + rows - 1) / d.T + 1;
    const int tt = tfirst + threadIdx.x, i = tt / d.T, t = tt - i * d.T;
    float p[13];
    if ((int)threadIdx.x < rows) {
      const int bh = bh0 + i, b = bh / d.H, h = bh - b * d.H;
      load_row13<T>(params + ((long long)b * d.T + t) * d.ps + (long long)h * 13, row13_wide(d, h), p);
    }
    for (int e = threadIdx.x; e < n_bh; e += 256) {
      const size_t at = (size_t)((bh0 + e) % d.H) * pp.bias_stride;
#pragma unroll
      for (int k = 0; k < 7; ++k) sbias[7 * e + k] = load_as_f(pp.bias[k], pp.dtype, at);
    }
    __syncthreads();
    if ((int)threadIdx.x < rows) {
      const long long row = row0 + threadIdx.x;
      const float *bi = sbias + 7 * i;
      p[0] += bi[0]; p[1] += bi[1]; p[2] += bi[2]; p[5] += bi[3]; p[6] += bi[4]; p[7] += bi[5]; p[8] += bi[6];
      const CoefOut o = coef_forward(p, hp, nullptr);
      *reinterpret_cast<float2 *>(M + row * 2) = o.rho;
      *reinterpret_cast<float4 *>(K + row * 4) = make_float4(o.kp.x, o.kp.y, o.kc.x, o.kc.y);
    }
  }

  // ---- the wide rows ----
  Walk cur{tfirst + grp, bh0, 0, 0};
  settle(cur);
  float sc[4][VEC];
  int sc_h = -1;
  const int n_iter = (rows + NG - 1) / NG;  // the same for every group: the shuffles below need whole warps
  for (int i = 0; i < n_iter; ++i) {
    request(i + kPrepRing - 1);  // into the slot read in the previous iteration
    copy_wait<kPrepRing - 1>();
    const bool live = grp + i * NG < rows;
    const uint4 *s = slot + (i % kPrepRing) * 5 * 256;
    const long long row = row0 + grp + (long long)i * NG;
    if (live && on_p) *reinterpret_cast<uint4 *>(U + row * d.P + n0) = s[4 * 256];
    uint4 raw[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) raw[j] = (live && on_n) ? s[j * 256] : make_uint4(0, 0, 0, 0);
    auto elem = [&](int j, int e) { return to_f(reinterpret_cast<const T *>(&raw[j])[e]); };
    float ss[4] = {1.f, 1.f, 1.f, 1.f};
    if (d.normalize) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < VEC; ++e) a = fmaf(elem(j, e), elem(j, e), a);
        ss[j] = a;
      }
      group_sum4<G>(ss, [&](float w) { return rsqrtf(w / (float)d.N + 1e-5f); });
      if (live && on_n && sc_h != cur.h) {
        sc_h = cur.h;
#pragma unroll
        for (int j = 0; j < 4; ++j) load_scale<VEC>(pp, sc_h, j, d.N, n0, sc[j]);
      }
    }
    if (live && on_n) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {  // B from planes 0, 1 and C from planes 2, 3, interleaved
        float o[2][VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          float re = elem(2 * m, e), im = elem(2 * m + 1, e);
          if (d.normalize) {
            re = (re * ss[2 * m]) * sc[2 * m][e];
            im = (im * ss[2 * m + 1]) * sc[2 * m + 1][e];
          }
          const int k = 2 * e;
          o[k / VEC][k % VEC] = re;
          o[(k + 1) / VEC][(k + 1) % VEC] = im;
        }
        T *dst = (m == 0 ? Bo : Co) + row * D + 2 * n0;
        store_vec<T, VEC>(dst, o[0]);
        store_vec<T, VEC>(dst + VEC, o[1]);
      }
    }
    if (live) advance(cur);
  }
  copy_wait<0>();
}

// Forward, any width and alignment (rows the kernel above does not cover).  Rows are ordered (b, h, t) so that a
// CTA's consecutive rows write contiguous output.  A group of G lanes handles one row; lane q of the group owns the
// state lanes n in [VEC*(q + G*k), VEC*(q + G*k) + VEC).
template <typename T, int VEC, int G>
__global__ void __launch_bounds__(256) scanprep_fwd_any_kernel(const T *__restrict__ value, const T *__restrict__ params,
                                                           const T *__restrict__ bc, PrepParams pp, T *__restrict__ U,
                                                           float *__restrict__ M, float *__restrict__ K,
                                                           T *__restrict__ Bo, T *__restrict__ Co, PrepDims d,
                                                           PrepHyper hp) {
  // A CTA pass covers 256 consecutive rows.  Phase 1: one row per THREAD for the
  // coefficient map (its ~500 scalar instructions then cost one issue slot per 32 rows
  // instead of one per row).  Phase 2: one row per lane group for the wide copies.
  constexpr int GPB = 256 / G;   // lane groups per CTA
  constexpr int RPG = 256 / GPB; // rows each group walks through per pass (= G)
  const int q = threadIdx.x % G;
  const int grp = threadIdx.x / G;
  const long long n_rows = (long long)d.batch * d.H * d.T;
  const int D = 2 * d.N;
  for (long long row0 = (long long)blockIdx.x * 256; row0 < n_rows; row0 += (long long)gridDim.x * 256) {
    {
      const long long row = row0 + threadIdx.x;
      if (row < n_rows) {
        const int t = (int)(row % d.T);
        const int h = (int)((row / d.T) % d.H);
        const int b = (int)(row / ((long long)d.T * d.H));
        float p[13];
        const T *pr = params + ((long long)b * d.T + t) * d.ps + (long long)h * 13;
        load_row13<T>(pr, row13_wide(d, h), p);
        add_bias13(pp, h, p);
        CoefOut o = coef_forward(p, hp, nullptr);
        *reinterpret_cast<float2 *>(M + row * 2) = o.rho;
        *reinterpret_cast<float4 *>(K + row * 4) = make_float4(o.kp.x, o.kp.y, o.kc.x, o.kc.y);
      }
    }
    // (b, h, t) of the group's first row by division once per pass, then by increment
    const long long grow0 = row0 + (long long)grp * RPG;
    int gt, gh, gb;
    {
      const long long r = grow0 < n_rows ? grow0 : 0;
      gt = (int)(r % d.T);
      gh = (int)((r / d.T) % d.H);
      gb = (int)(r / ((long long)d.T * d.H));
    }
    for (int k = 0; k < RPG; ++k) {
      const long long row = grow0 + k;
      const bool live = row < n_rows;
      const long long rr = live ? row : 0;
      const int t = live ? gt : 0, h = live ? gh : 0, b = live ? gb : 0;
      // advance (b, h, t) to the next row
      if (++gt == d.T) {
        gt = 0;
        if (++gh == d.H) {
          gh = 0;
          ++gb;
        }
      }
      const long long in_row = (long long)b * d.T + t;
      // ---- U: copy P values ----
      if (live) {
        const T *src = value + in_row * d.vs + (long long)h * d.P;
        T *dst = U + rr * d.P;
        for (int p0 = q * VEC; p0 < d.P; p0 += G * VEC) {
          float v[VEC];
          load_vec<T, VEC>(src + p0, v);
          store_vec<T, VEC>(dst + p0, v);
        }
      }
      // ---- B, C ----
      const T *bcr = bc + in_row * d.bs + (long long)h * 4 * d.N;
      float ss[4] = {0.f, 0.f, 0.f, 0.f};
      if (d.normalize) {
        if (live) {
          for (int n0 = q * VEC; n0 < d.N; n0 += G * VEC) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v[VEC];
              load_vec<T, VEC>(bcr + j * d.N + n0, v);
#pragma unroll
              for (int i = 0; i < VEC; ++i) ss[j] = fmaf(v[i], v[i], ss[j]);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) ss[j] = rsqrtf(group_sum_f<G>(ss[j]) / (float)d.N + 1e-5f);
      }
      if (live) {
        for (int n0 = q * VEC; n0 < d.N; n0 += G * VEC) {
          float y[4][VEC];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            load_vec<T, VEC>(bcr + j * d.N + n0, y[j]);
            if (d.normalize) {
              float sc[VEC];
              load_scale<VEC>(pp, h, j, d.N, n0, sc);
#pragma unroll
              for (int i = 0; i < VEC; ++i) y[j][i] = (y[j][i] * ss[j]) * sc[i];
            }
          }
          float ob[2][VEC], oc[2][VEC];
#pragma unroll
          for (int i = 0; i < VEC; ++i) {
            int o = 2 * i;
            ob[o / VEC][o % VEC] = y[0][i];
            ob[(o + 1) / VEC][(o + 1) % VEC] = y[1][i];
            oc[o / VEC][o % VEC] = y[2][i];
            oc[(o + 1) / VEC][(o + 1) % VEC] = y[3][i];
          }
          store_vec<T, VEC>(Bo + rr * D + 2 * n0, ob[0]);
          store_vec<T, VEC>(Bo + rr * D + 2 * n0 + VEC, ob[1]);
          store_vec<T, VEC>(Co + rr * D + 2 * n0, oc[0]);
          store_vec<T, VEC>(Co + rr * D + 2 * n0 + VEC, oc[1]);
        }
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void scanprep_bwd_coef_tile(const T *__restrict__ params, const PrepParams &pp,
                                                       const float *__restrict__ dM, const float *__restrict__ dK,
                                                       T *__restrict__ d_params, float *__restrict__ part,
                                                       const PrepDims &d, const PrepHyper &hp, int rows_per_tile,
                                                       int tile, int n_tiles);

// Backward, rows that one 16-byte slice per lane covers (as scanprep_fwd_kernel).  Reads nine slices per lane and row
// (bc, dB, dC, dU), writes five.  grid = (2 * tiles over T, batch*H): the first half of a row of CTAs streams the wide
// rows, the second runs the coefficient-map VJP of the same tiles, whose long scalar chains fill issue slots that
// the streaming CTAs leave (run inside the streaming CTAs ahead of their rows it cost a third of the kernel's time).
// A CTA works on one head, so that the parameter gradients reduce inside it first (registers, then shared memory in
// a fixed order) and across CTAs in a second kernel.
// HBM bounds the traffic, but the arithmetic on 64 values per lane and row is nearly as long: it works on (re, im)
// pairs with two-wide fp32 instructions.  With r = 1/rms the two row sums, sum x^2 and sum g x (g = scale dy), are
// taken together before r exists, so that the group synchronises once; then
//   d_scale += dy x r,   dx = r g - x r^3 (sum g x) / N.
// b16 T4096 16 heads N128: 0.707 ms (0.78 of the copy rate; 0.770 with rows requested when needed, 16 lanes per row and
// 8-byte slices unless everything is 16-byte aligned); b8 T2048 12 heads N64: 0.101 ms (0.195).
// Partial layout: part[(bh * n_tiles + tile)][4*N + 13].
constexpr int kPrepBwdSlices = 9;
#define SLX_OPAQUE4(u) asm volatile("" : "+r"((u).x), "+r"((u).y), "+r"((u).z), "+r"((u).w))
template <typename T, int VEC, int G, int AL>
__global__ void __launch_bounds__(256, 2) scanprep_bwd_kernel(const T *__restrict__ params, const T *__restrict__ bc,
                                                              PrepParams pp, const T *__restrict__ dU,
                                                              const float *__restrict__ dM,
                                                              const float *__restrict__ dK, const T *__restrict__ dB,
                                                              const T *__restrict__ dC, T *__restrict__ d_value,
                                                              T *__restrict__ d_params, T *__restrict__ d_bc,
                                                              float *__restrict__ part, PrepDims d, PrepHyper hp,
                                                              int rows_per_tile, int n_tiles) {
  if ((int)blockIdx.x >= n_tiles) {
    scanprep_bwd_coef_tile<T>(params, pp, dM, dK, d_params, part, d, hp, rows_per_tile, (int)blockIdx.x - n_tiles,
                              n_tiles);
    return;
  }
  constexpr int NG = 256 / G;
  extern __shared__ uint4 prep_ring[];  // [kPrepRing][9][256 threads] (afterwards the groups' d_scale sums), scales
  // scale of the head as (re, im) pairs, two neighbouring state lanes per 16 bytes, laid out
  // [B, C][VEC / 2][G lanes]: a warp reads consecutive 16-byte words
  float4 *sscale = reinterpret_cast<float4 *>(prep_ring + kPrepRing * kPrepBwdSlices * 256);
  const int q = threadIdx.x % G, grp = threadIdx.x / G;
  const int n0 = q * VEC;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  const int D = 2 * d.N, W = 4 * d.N + 13;
  const int t_lo = blockIdx.x * rows_per_tile, rows = min(d.T - t_lo, rows_per_tile);
  const bool on_n = n0 < d.N, on_p = n0 < d.P;
  const long long in0 = (long long)b * d.T + t_lo, out0 = (long long)bh * d.T + t_lo;
  uint4 *slot = prep_ring + threadIdx.x;
  auto request = [&](int i) {  // row grp + i * NG of the tile into ring slot i % kPrepRing
    const int r = grp + i * NG;
    if (r < rows) {
      uint4 *s = slot + (i % kPrepRing) * kPrepBwdSlices * 256;
      if (on_n) {
        const T *x = bc + (in0 + r) * d.bs + (long long)h * 4 * d.N + n0;
        const T *gb = dB + (out0 + r) * D + 2 * n0, *gc = dC + (out0 + r) * D + 2 * n0;
#pragma unroll
        for (int j = 0; j < 4; ++j) copy_slice<AL>(s + j * 256, x + j * d.N);
        copy_slice<16>(s + 4 * 256, gb);
        copy_slice<16>(s + 5 * 256, gb + VEC);
        copy_slice<16>(s + 6 * 256, gc);
        copy_slice<16>(s + 7 * 256, gc + VEC);
      }
      if (on_p) copy_slice<16>(s + 8 * 256, dU + (out0 + r) * d.P + n0);
    }
    copy_commit();
  };
#pragma unroll
  for (int i = 0; i < kPrepRing - 1; ++i) request(i);

  if (d.normalize) {
    for (int w = threadIdx.x; w < VEC * G; w += 256) {
      const int m = w / (VEC / 2 * G), n = w % G * VEC + w / G % (VEC / 2) * 2;  // lanes n, n + 1
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (n < d.N) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          v[k] = load_as_f(scale_plane(pp, 2 * m), pp.dtype, scale_index(pp, h, 2 * m + (k & 1), d.N, n + (k >> 1)));
      }
      sscale[w] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
  }
  float2 dsc[2][VEC];  // [B, C][lane]: (re, im)
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int e = 0; e < VEC; ++e) dsc[m][e] = make_float2(0.f, 0.f);
  const float inv_n = 1.f / (float)d.N;
  const int n_iter = (rows + NG - 1) / NG;
  for (int i = 0; i < n_iter; ++i) {
    request(i + kPrepRing - 1);
    copy_wait<kPrepRing - 1>();
    const int r = grp + i * NG;
    const bool live = r < rows, mine = live && on_n;
    const uint4 *s = slot + (i % kPrepRing) * kPrepBwdSlices * 256;
    if (live && on_p)
      *reinterpret_cast<uint4 *>(d_value + (in0 + r) * ((long long)d.H * d.P) + (long long)h * d.P + n0) = s[8 * 256];
    T *dst = d_bc + (in0 + r) * ((long long)d.H * 4 * d.N) + (long long)h * 4 * d.N + n0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {  // B, then C: half the row's registers at a time (all of it spilled)
      uint4 xr[2], gr[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        xr[j] = mine ? s[(2 * m + j) * 256] : make_uint4(0, 0, 0, 0);
        gr[j] = mine ? s[(4 + 2 * m + j) * 256] : make_uint4(0, 0, 0, 0);
      }
      // (re, im) of lane e: x from two planes, dy as it lies
      auto x_of = [&](int e) {
        return make_float2(to_f(reinterpret_cast<const T *>(&xr[0])[e]), to_f(reinterpret_cast<const T *>(&xr[1])[e]));
      };
      auto dy_of = [&](int e) {
        const T *g = reinterpret_cast<const T *>(&gr[2 * e / VEC]) + 2 * e % VEC;
        return make_float2(to_f(g[0]), to_f(g[1]));
      };
      auto sc_of = [&](int e) {
        const float4 v = sscale[(m * (VEC / 2) + e / 2) * G + q];
        return e & 1 ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
      };
      float o[2][VEC];
      if (d.normalize) {
        float2 a = make_float2(0.f, 0.f), c = a;
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float2 x = x_of(e);
          a = __ffma2_rn(x, x, a);
          c = __ffma2_rn(__fmul2_rn(dy_of(e), sc_of(e)), x, c);
        }
        // the packed words stay opaque across the shuffles: expanding them again is a few shifts, holding the
        // expanded values spilled
        SLX_OPAQUE4(xr[0]);
        SLX_OPAQUE4(xr[1]);
        SLX_OPAQUE4(gr[0]);
        SLX_OPAQUE4(gr[1]);
        float v[4] = {a.x, a.y, c.x, c.y};
        const bool is_square = !(threadIdx.x & 1);  // which of the four sums this lane finishes (group_sum4)
        group_sum4<G>(v, [&](float w) { return is_square ? rsqrtf(w * inv_n + 1e-5f) : w * inv_n; });
        const float2 rs = make_float2(v[0], v[1]);
        // (r v first: r^3 alone leaves the range of fp32 for rows of magnitude 1e13)
        const float2 cc = make_float2(-(rs.x * v[2]) * (rs.x * rs.x), -(rs.y * v[3]) * (rs.y * rs.y));
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float2 x = x_of(e), dy = dy_of(e);
          dsc[m][e] = __ffma2_rn(__fmul2_rn(dy, x), rs, dsc[m][e]);
          const float2 dx = __ffma2_rn(x, cc, __fmul2_rn(rs, __fmul2_rn(dy, sc_of(e))));
          o[0][e] = dx.x;
          o[1][e] = dx.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float2 dy = dy_of(e);
          o[0][e] = dy.x;
          o[1][e] = dy.y;
        }
      }
      if (mine) {
        store_vec<T, VEC>(dst + 2 * m * d.N, o[0]);
        store_vec<T, VEC>(dst + (2 * m + 1) * d.N, o[1]);
      }
      asm volatile("" ::: "memory");
    }
  }
  copy_wait<0>();
  __syncthreads();  // every lane is done with its ring slots: the ring becomes the groups' sums
  float *red = reinterpret_cast<float *>(prep_ring);  // [NG][4N]
  if (on_n) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        red[(size_t)grp * 4 * d.N + 2 * m * d.N + n0 + e] = dsc[m][e].x;
        red[(size_t)grp * 4 * d.N + (2 * m + 1) * d.N + n0 + e] = dsc[m][e].y;
      }
  }
  __syncthreads();
  float *outp = part + ((size_t)bh * n_tiles + blockIdx.x) * W;
  for (int e = threadIdx.x; e < 4 * d.N; e += 256) {  // (the 13 bias slots are written by the coefficient CTAs)
    float acc = 0.f;
    for (int g = 0; g < NG; ++g) acc += red[(size_t)g * 4 * d.N + e];
    outp[e] = acc;
  }
}

// Backward, any width and alignment.  grid = (2 * tiles over T, batch*H).  CTAs with blockIdx.x < n_tiles stream the
// wide rows; the others run the coefficient-map VJP of the same tiles.  Same partial layout.
template <typename T, int VEC, int G, int KMAX>
__global__ void __launch_bounds__(256, KMAX == 1 ? 2 : 1) scanprep_bwd_any_kernel(const T *__restrict__ params, const T *__restrict__ bc,
                                                           PrepParams pp, const T *__restrict__ dU,
                                                           const float *__restrict__ dM, const float *__restrict__ dK,
                                                           const T *__restrict__ dB, const T *__restrict__ dC,
                                                           T *__restrict__ d_value, T *__restrict__ d_params,
                                                           T *__restrict__ d_bc, float *__restrict__ part, PrepDims d,
                                                           PrepHyper hp, int rows_per_tile, int n_tiles) {
  if ((int)blockIdx.x >= n_tiles) {
    scanprep_bwd_coef_tile<T>(params, pp, dM, dK, d_params, part, d, hp, rows_per_tile, (int)blockIdx.x - n_tiles,
                              n_tiles);
    return;
  }
  constexpr int GPB = 256 / G;  // KMAX sweeps of VEC*G state lanes cover N
  extern __shared__ float red[];  // GPB * (4N + 13)
  const int q = threadIdx.x % G, grp = threadIdx.x / G;
  const int bh = blockIdx.y, b = bh / d.H, h = bh % d.H;
  const int D = 2 * d.N;
  const int W = 4 * d.N + 13;
  const int t_lo = blockIdx.x * rows_per_tile;
  const int t_hi = min(d.T, t_lo + rows_per_tile);

  float dsc[KMAX][4][VEC];
#pragma unroll
  for (int k = 0; k < KMAX; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < VEC; ++i) dsc[k][j][i] = 0.f;
  for (int tb = t_lo; tb < t_hi; tb += GPB) {
    const int t = tb + grp;
    const bool live = t < t_hi;
    const int tt = live ? t : t_lo;
    const long long in_row = (long long)b * d.T + tt;
    const long long orow = ((long long)bh) * d.T + tt;
    if (live) {
      const T *src = dU + orow * d.P;
      T *dst = d_value + in_row * ((long long)d.H * d.P) + (long long)h * d.P;
      for (int p0 = q * VEC; p0 < d.P; p0 += G * VEC) {
        float v[VEC];
        load_vec<T, VEC>(src + p0, v);
        store_vec<T, VEC>(dst + p0, v);
      }
    }
    const T *bcr = bc + in_row * d.bs + (long long)h * 4 * d.N;
    T *dbcr = d_bc + in_row * ((long long)d.H * 4 * d.N) + (long long)h * 4 * d.N;
    float ss[4] = {0.f, 0.f, 0.f, 0.f}, gx[4] = {0.f, 0.f, 0.f, 0.f};
    if (d.normalize) {
      if (live) {
        int k = 0;
        for (int n0 = q * VEC; n0 < d.N; n0 += G * VEC, ++k) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v[VEC];
            load_vec<T, VEC>(bcr + j * d.N + n0, v);
#pragma unroll
            for (int i = 0; i < VEC; ++i) ss[j] = fmaf(v[i], v[i], ss[j]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) ss[j] = rsqrtf(group_sum_f<G>(ss[j]) / (float)d.N + 1e-5f);
    }
    // second sweep: dy (de-interleaved), dscale, sum g*xhat
    float xh[KMAX][4][VEC], gg[KMAX][4][VEC];
    {
      int k = 0;
      for (int n0 = q * VEC; n0 < d.N && k < KMAX; n0 += G * VEC, ++k) {
        float ib[2][VEC], ic[2][VEC];
        if (live) {
          load_vec<T, VEC>(dB + orow * D + 2 * n0, ib[0]);
          load_vec<T, VEC>(dB + orow * D + 2 * n0 + VEC, ib[1]);
          load_vec<T, VEC>(dC + orow * D + 2 * n0, ic[0]);
          load_vec<T, VEC>(dC + orow * D + 2 * n0 + VEC, ic[1]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x[VEC];
          if (live) load_vec<T, VEC>(bcr + j * d.N + n0, x);
#pragma unroll
          for (int i = 0; i < VEC; ++i) {
            int o = 2 * i + (j & 1);
            float dy = 0.f;
            if (live) dy = (j < 2) ? ib[o / VEC][o % VEC] : ic[o / VEC][o % VEC];
            if (d.normalize) {
              float xv = live ? x[i] * ss[j] : 0.f;
              float g = dy * load_as_f(scale_plane(pp, j), pp.dtype, scale_index(pp, h, j, d.N, n0 + i));
              xh[k][j][i] = xv;
              gg[k][j][i] = g;
              dsc[k][j][i] = fmaf(dy, xv, dsc[k][j][i]);
              gx[j] = fmaf(g, xv, gx[j]);
            } else {
              gg[k][j][i] = dy;
            }
          }
        }
      }
    }
    if (d.normalize) {
#pragma unroll
      for (int j = 0; j < 4; ++j) gx[j] = group_sum_f<G>(gx[j]) / (float)d.N;
    }
    if (live) {
      int k = 0;
      for (int n0 = q * VEC; n0 < d.N && k < KMAX; n0 += G * VEC, ++k) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float o[VEC];
#pragma unroll
          for (int i = 0; i < VEC; ++i)
            o[i] = d.normalize ? ss[j] * (gg[k][j][i] - xh[k][j][i] * gx[j]) : gg[k][j][i];
          store_vec<T, VEC>(dbcr + j * d.N + n0, o);
        }
      }
    }
  }
  // ---- CTA-level reduction in a fixed order ----
  {
    float *mine = red + (size_t)grp * W;
    if (d.normalize) {
      int k = 0;
      for (int n0 = q * VEC; n0 < d.N && k < KMAX; n0 += G * VEC, ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < VEC; ++i) mine[j * d.N + n0 + i] = dsc[k][j][i];
    }
  }
  __syncthreads();
  float *outp = part + ((size_t)bh * n_tiles + blockIdx.x) * W;
  for (int e = threadIdx.x; e < W; e += 256) {
    if (!d.normalize && e < 4 * d.N) {
      outp[e] = 0.f;
      continue;
    }
    if (e >= 4 * d.N) continue;  // the 13 bias slots belong to the coefficient CTAs
    float acc = 0.f;
    for (int g = 0; g < GPB; ++g) acc += red[(size_t)g * W + e];
    outp[e] = acc;
  }
}

// Coefficient-map VJP of the backward: one row per thread (rows_per_tile == blockDim.x),
// d_params rows and the per-tile partial sums of the 13 bias gradients
// (part[(bh * n_tiles + tile)][4N .. 4N+13)).  Little traffic, long scalar chains.
template <typename T>
__device__ __forceinline__ void scanprep_bwd_coef_tile(const T *__restrict__ params, const PrepParams &pp,
                                                       const float *__restrict__ dM, const float *__restrict__ dK,
                                                       T *__restrict__ d_params, float *__restrict__ part,
                                                       const PrepDims &d, const PrepHyper &hp, int rows_per_tile,
                                                       int tile, int n_tiles) {
  const int bh = blockIdx.y, b = bh / d.H, h = bh % d.H;
  const int W = 4 * d.N + 13;
  const int t_lo = tile * rows_per_tile;
  const int t_hi = min(d.T, t_lo + rows_per_tile);
  __shared__ float sbias[8][13];
  {
    float dbias[13];
#pragma unroll
    for (int i = 0; i < 13; ++i) dbias[i] = 0.f;
    for (int t = t_lo + (int)threadIdx.x; t < t_hi; t += 256) {
      const long long in_row = (long long)b * d.T + t;
      const long long orow = ((long long)bh) * d.T + t;
      float p[13], dp[13];
      const T *pr = params + in_row * d.ps + (long long)h * 13;
      load_row13<T>(pr, row13_wide(d, h), p);
      add_bias13(pp, h, p);
      CoefCtx ctx;
      coef_forward(p, hp, &ctx);
      float2 dm = *reinterpret_cast<const float2 *>(dM + orow * 2);
      float4 dk = *reinterpret_cast<const float4 *>(dK + orow * 4);
      coef_backward(ctx, hp, dm, make_float2(dk.x, dk.y), make_float2(dk.z, dk.w), dp);
      store_row13<T>(d_params + in_row * ((long long)d.H * 13) + (long long)h * 13, dp);
#pragma unroll
      for (int i = 0; i < 13; ++i) dbias[i] += dp[i];
    }
#pragma unroll
    for (int i = 0; i < 13; ++i) {
      float v = dbias[i];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if ((threadIdx.x & 31) == 0) sbias[threadIdx.x >> 5][i] = v;
    }
  }

  __syncthreads();
  if (threadIdx.x < 13) {
    float acc = 0.f;
    for (int w = 0; w < 8; ++w) acc += sbias[w][threadIdx.x];
    part[((size_t)bh * n_tiles + tile) * W + 4 * d.N + threadIdx.x] = acc;
  }
}

// d_scale[h][e], d_bias[h][i] = sum over batch and tiles of the partials, fixed order
struct PrepParamGrads {
  float *bias13;                // [opt] (H,13) fp32, every slot
  void *bias[7];                // [opt] the seven biases' gradients, H values each, as dtype
  void *b_scale, *c_scale;      // [opt] as dtype, laid out like the parameters (scale_stride per head)
  int dtype;
  long long scale_stride;
};
__global__ void scanprep_reduce_kernel(const float *__restrict__ part, PrepParamGrads g, int batch, int H, int n_tiles,
                                       int N) {
  const int W = 4 * N + 13;
  const int h = blockIdx.y;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= W) return;
  float acc = 0.f;
  for (int b = 0; b < batch; ++b) {
    const float *pb = part + ((size_t)(b * H + h) * n_tiles) * W + e;
    int tile = 0;
    for (; tile + 8 <= n_tiles; tile += 8) {  // eight loads in flight, summed in the fixed order
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = pb[(size_t)(tile + i) * W];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc += v[i];
    }
    for (; tile < n_tiles; ++tile) acc += pb[(size_t)tile * W];
  }
  if (e < 4 * N) {
    const int j = e / N, n = e - j * N;
    void *base = j < 2 ? g.b_scale : g.c_scale;
    if (base) store_as(base, g.dtype, (size_t)h * g.scale_stride + (size_t)(j & 1) * N + n, acc);
  } else {
    const int slot = e - 4 * N;
    if (g.bias13) g.bias13[h * 13 + slot] = acc;
    const int k = slot < 3 ? slot : (slot >= 5 && slot < 9 ? slot - 2 : -1);
    if (k >= 0 && g.bias[k]) store_as(g.bias[k], g.dtype, h, acc);
  }
}

static PrepHyper make_hyper(const slx_prep_shape *s) {
  PrepHyper h;
  h.dt_min = s->dt_min; h.dt_max = s->dt_max; h.r_min = s->r_min; h.r_max = s->r_max;
  h.theta_bound = s->theta_bound; h.k_max = s->k_max;
  float e = s->eps > 1e-12f ? s->eps : 1e-12f;
  float thr = sqrtf(e);
  if (thr < 1e-4f) thr = 1e-4f;
  h.z_thr2 = thr * thr;
  return h;
}

static int check_prep(const slx_prep_shape *s, PrepDims *d) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  SLX_REQUIRE(s->batch > 0 && s->T > 0 && s->heads > 0 && s->P > 0 && s->N > 0, SLX_E_SHAPE,
              "scanprep: sizes must be positive");
  SLX_REQUIRE(s->dtype >= SLX_F32 && s->dtype <= SLX_F16, SLX_E_DTYPE, "scanprep: bad dtype %d", s->dtype);
  SLX_REQUIRE(s->value_stride >= (int64_t)s->heads * s->P && s->params_stride >= (int64_t)s->heads * 13 &&
                  s->bc_stride >= (int64_t)s->heads * 4 * s->N,
              SLX_E_SHAPE, "scanprep: row stride smaller than the row width");
  SLX_REQUIRE((long long)s->batch * s->heads <= 65535, SLX_E_UNSUPPORTED, "scanprep: batch*heads exceeds 65535");
  d->batch = s->batch; d->T = s->T; d->H = s->heads; d->P = s->P; d->N = s->N;
  d->normalize = s->normalize_bc;
  d->vs = s->value_stride; d->ps = s->params_stride; d->bs = s->bc_stride;
  d->wide_params = 0;
  return SLX_OK;
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// params rows of a half type that start on 16-byte boundaries: a head's 13 values can be picked out of the aligned
// vectors that cover them (row13_wide says for which heads those lie inside the row)
static int params_rows_wide(const slx_prep_shape *s, const void *params) {
  return s->dtype != SLX_F32 && aligned16(params) && (s->params_stride * 2) % 16 == 0;
}

// vector width (elements) usable for this problem: 16-byte vectors when every row start and row
// width is 16-byte aligned, 8-byte vectors when they are 8-byte aligned (a projection whose row
// is a multiple of 4 but not of 8 half values, e.g. 4764 = 2*768 + 12*13 + 4*12*64), else scalar
template <typename T>
static int pick_vec(const slx_prep_shape *s, std::initializer_list<const void *> ptrs) {
  for (int bytes = 16; bytes >= 8; bytes /= 2) {
    const int v = bytes / (int)sizeof(T);
    bool ok = (s->N % v == 0) && (s->P % v == 0) && (s->value_stride % v == 0) && (s->bc_stride % v == 0);
    for (const void *p : ptrs) ok = ok && (p == nullptr || (reinterpret_cast<uintptr_t>(p) % bytes) == 0);
    if (ok) return v;
  }
  return 1;
}

// lane-group width: 16 lanes x 16-byte vectors cover N = 128 half values in one
// sweep; the scalar mapping uses a full warp per row
template <int VEC>
constexpr int prep_group() { return VEC == 1 ? 32 : 16; }

template <typename T, int VEC>
static int launch_prep_fwd_any(const slx_prep_shape *s, const PrepDims &d, const void *value, const void *params,
                               const void *bc, const PrepParams &pp, void *U, float *M, float *K, void *B, void *C,
                               cudaStream_t st) {
  PrepHyper hp = make_hyper(s);
  constexpr int G = prep_group<VEC>();
  long long n_rows = (long long)d.batch * d.H * d.T;
  long long blocks = (n_rows + 255) / 256;
  if (blocks > kB200Sms * 32LL) blocks = kB200Sms * 32LL;
  scanprep_fwd_any_kernel<T, VEC, G><<<(unsigned)blocks, 256, 0, st>>>(
      (const T *)value, (const T *)params, (const T *)bc, pp, (T *)U, M, K, (T *)B, (T *)C, d, hp);
  return check_launch("scanprep_fwd");
}

// Rows per CTA of the one-slice forward: as many as make the grid whole waves of three CTAs per SM, at most 256 (one
// per thread in the coefficient map), at least 32.
static int prep_rows_per_cta(long long n_rows) {
  const long long slots = kB200Sms * 3LL, waves = (n_rows + slots * 256 - 1) / (slots * 256);
  long long r = (n_rows + slots * waves - 1) / (slots * waves);
  r = (r + 7) / 8 * 8;
  return (int)(r < 32 ? 32 : r);
}
template <typename T, int G, int AL>
static int launch_prep_fwd(const slx_prep_shape *s, const PrepDims &d, const void *value, const void *params,
                           const void *bc, const PrepParams &pp, void *U, float *M, float *K, void *B, void *C,
                           cudaStream_t st) {
  constexpr size_t ring = (size_t)kPrepRing * 5 * 256 * 16;
  auto kern = scanprep_fwd_kernel<T, 16 / (int)sizeof(T), G, AL>;
  int rc = ensure_dyn_smem(kern, ring);
  if (rc) return rc;
  const long long n_rows = (long long)d.batch * d.H * d.T;
  const int rows = prep_rows_per_cta(n_rows);
  kern<<<(unsigned)((n_rows + rows - 1) / rows), 256, ring, st>>>((const T *)value, (const T *)params, (const T *)bc, pp,
                                                                 (T *)U, M, K, (T *)B, (T *)C, d, make_hyper(s), rows);
  return check_launch("scanprep_fwd");
}
template <typename T, int AL, typename... A>
static int launch_prep_fwd_lanes(int lanes, const A &...args) {
  switch (lanes) {
    case 4: return launch_prep_fwd<T, 4, AL>(args...);
    case 8: return launch_prep_fwd<T, 8, AL>(args...);
    case 16: return launch_prep_fwd<T, 16, AL>(args...);
    default: return launch_prep_fwd<T, 32, AL>(args...);
  }
}
// lanes per row of the one-slice kernels (0: the row is wider than a warp's slices)
template <typename T>
static int prep_lanes(const slx_prep_shape *s) {
  constexpr int v = 16 / (int)sizeof(T);
  const int need = ((s->N > s->P ? s->N : s->P) + v - 1) / v;
  return need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : need <= 32 ? 32 : 0;
}

struct PrepBwdPlan {
  int G, kmax, rows_per_tile, n_tiles;
  size_t smem, ws_bytes;
};

static PrepBwdPlan prep_bwd_plan(const slx_prep_shape *s, int VEC) {
  PrepBwdPlan p;
  p.G = VEC == 1 ? 32 : 16;
  p.kmax = (s->N + VEC * p.G - 1) / (VEC * p.G);
  // Tiles of at most 256 rows (one per thread in the coefficient part), as many as make whole waves of two CTAs per
  // SM, of 32 rows at least.
  const long long slots = kB200Sms * 2LL, bh = (long long)s->batch * s->heads;
  const long long waves = (bh * ((s->T + 255) / 256) + slots - 1) / slots;
  long long n = waves * slots / bh;
  if (n < (s->T + 255) / 256) n = (s->T + 255) / 256;
  long long r = ((s->T + n - 1) / n + 7) / 8 * 8;
  p.rows_per_tile = (int)(r < 32 ? 32 : r > 256 ? 256 : r);
  p.n_tiles = (s->T + p.rows_per_tile - 1) / p.rows_per_tile;
  int W = 4 * s->N + 13;
  p.smem = sizeof(float) * (size_t)(256 / p.G) * W;  // group partials (any-width kernel)
  p.ws_bytes = sizeof(float) * (size_t)s->batch * s->heads * p.n_tiles * W;
  return p;
}

template <typename T>
static int launch_prep_reduce(const PrepDims &d, const float *part, const PrepParamGrads &pg, int n_tiles,
                              cudaStream_t st) {
  const int W = 4 * d.N + 13;
  scanprep_reduce_kernel<<<dim3((W + 127) / 128, d.H), 128, 0, st>>>(part, pg, d.batch, d.H, n_tiles, d.N);
  return check_launch("scanprep_reduce");
}

template <typename T, int G, int AL>
static int launch_prep_bwd_rows(const slx_prep_shape *s, const PrepDims &d, const void *params, const void *bc,
                                const PrepParams &pp, const void *dU, const float *dM, const float *dK, const void *dB,
                                const void *dC, void *d_value, void *d_params, void *d_bc, const PrepParamGrads &pg,
                                float *part, cudaStream_t st) {
  constexpr int VEC = 16 / (int)sizeof(T);
  const PrepBwdPlan pl = prep_bwd_plan(s, VEC);
  const size_t smem = (size_t)kPrepRing * kPrepBwdSlices * 256 * 16 + (size_t)VEC * G * 16;
  static_assert((size_t)kPrepRing * kPrepBwdSlices * 256 * 16 >= sizeof(float) * 256 * 4 * VEC, "d_scale sums fit the ring");
  auto kern = scanprep_bwd_kernel<T, VEC, G, AL>;
  int rc = ensure_dyn_smem(kern, smem);
  if (rc) return rc;
  kern<<<dim3(2 * pl.n_tiles, d.batch * d.H), 256, smem, st>>>(
      (const T *)params, (const T *)bc, pp, (const T *)dU, dM, dK, (const T *)dB, (const T *)dC, (T *)d_value,
      (T *)d_params, (T *)d_bc, part, d, make_hyper(s), pl.rows_per_tile, pl.n_tiles);
  rc = check_launch("scanprep_bwd");
  return rc ? rc : launch_prep_reduce<T>(d, part, pg, pl.n_tiles, st);
}
template <typename T, int AL, typename... A>
static int launch_prep_bwd_lanes(int lanes, const A &...args) {
  switch (lanes) {
    case 4: return launch_prep_bwd_rows<T, 4, AL>(args...);
    case 8: return launch_prep_bwd_rows<T, 8, AL>(args...);
    case 16: return launch_prep_bwd_rows<T, 16, AL>(args...);
    default: return launch_prep_bwd_rows<T, 32, AL>(args...);
  }
}

template <typename T, int VEC>
static int launch_prep_bwd(const slx_prep_shape *s, const PrepDims &d, const void *params, const void *bc,
                           const PrepParams &pp, const void *dU, const float *dM, const float *dK,
                           const void *dB, const void *dC, void *d_value, void *d_params, void *d_bc,
                           const PrepParamGrads &pg, float *part, cudaStream_t st) {
  PrepHyper hp = make_hyper(s);
  PrepBwdPlan pl = prep_bwd_plan(s, VEC);
  SLX_REQUIRE(pl.kmax <= 4, SLX_E_UNSUPPORTED, "scanprep_bwd: N=%d too large for the lane mapping", d.N);
  SLX_REQUIRE(pl.smem <= 200 * 1024, SLX_E_UNSUPPORTED, "scanprep_bwd: N=%d needs too much shared memory", d.N);
  constexpr int G = prep_group<VEC>();
#define SLX_PREP_BWD(KM)                                                                                      \
  {                                                                                                           \
    auto kern = scanprep_bwd_any_kernel<T, VEC, G, KM>;                                                           \
    int rc_smem = ensure_dyn_smem(kern, pl.smem);                                                             \
    if (rc_smem) return rc_smem;                                                                              \
    kern<<<dim3(2 * pl.n_tiles, d.batch * d.H), 256, pl.smem, st>>>(                                          \
        (const T *)params, (const T *)bc, pp, (const T *)dU, dM, dK, (const T *)dB, (const T *)dC,   \
        (T *)d_value, (T *)d_params, (T *)d_bc, part, d, hp, pl.rows_per_tile, pl.n_tiles);                   \
  }
  if (pl.kmax <= 1) SLX_PREP_BWD(1)
  else if (pl.kmax == 2) SLX_PREP_BWD(2)
  else SLX_PREP_BWD(4)
#undef SLX_PREP_BWD
  int rc = check_launch("scanprep_bwd");
  return rc ? rc : launch_prep_reduce<T>(d, part, pg, pl.n_tiles, st);
}

}  // namespace slx

using namespace slx;

#define SLX_PREP_T(dt, ...)                                          \
  switch (dt) {                                                      \
    case SLX_F32: { using T_ = float; __VA_ARGS__; } break;          \
    case SLX_BF16: { using T_ = __nv_bfloat16; __VA_ARGS__; } break; \
    default: { using T_ = __half; __VA_ARGS__; } break;              \
  }

static PrepParams f32_prep_params(const slx_prep_shape *s, const float *bias, const float *scale) {
  constexpr int kSlot[7] = {0, 1, 2, 5, 6, 7, 8};
  PrepParams pp{};
  for (int k = 0; k < 7; ++k) pp.bias[k] = bias ? bias + kSlot[k] : nullptr;
  pp.b_scale = scale;
  pp.c_scale = scale ? scale + 2 * s->N : nullptr;
  pp.dtype = SLX_F32;
  pp.bias_stride = 13;
  pp.scale_stride = 4LL * s->N;
  return pp;
}
static int make_prep_params(const slx_prep_shape *s, const slx_prep_params *p, PrepParams *pp) {
  SLX_REQUIRE(p != nullptr, SLX_E_NULL, "scanprep: params is NULL");
  SLX_REQUIRE(p->dtype >= SLX_F32 && p->dtype <= SLX_F16, SLX_E_DTYPE, "scanprep: bad parameter dtype %d", p->dtype);
  for (int k = 0; k < 7; ++k) {
    SLX_REQUIRE(p->bias[k] != nullptr, SLX_E_NULL, "scanprep: bias %d is NULL", k);
    pp->bias[k] = p->bias[k];
  }
  SLX_REQUIRE(!s->normalize_bc || (p->b_scale && p->c_scale), SLX_E_NULL, "scanprep: scale is NULL with normalize_bc set");
  pp->b_scale = p->b_scale;
  pp->c_scale = p->c_scale;
  pp->dtype = p->dtype;
  pp->bias_stride = 1;
  pp->scale_stride = 2LL * s->N;
  return SLX_OK;
}

static int prep_fwd_impl(const slx_prep_shape *s, const void *value, const void *params, const void *bc,
                         const PrepParams &pp, void *U, float *M, float *K, void *B, void *C, void *stream) {
  PrepDims d;
  int rc = check_prep(s, &d);
  if (rc) return rc;
  SLX_REQUIRE(value && params && bc && U && M && K && B && C, SLX_E_NULL, "scanprep_fwd: NULL tensor");
  d.wide_params = params_rows_wide(s, params);
  cudaStream_t st = as_stream(stream);
  SLX_PREP_T(s->dtype, {
    constexpr int VFULL = 16 / (int)sizeof(T_);
    const int G = prep_lanes<T_>(s);
    // 16-byte slices need N and P in whole slices, rows and pointers aligned to 16 bytes or (copied as two halves) 8:
    // a projection row of 4 but not 8 half values' multiple, e.g. 2*768 + 12*13 in front of bc
    int al = 0;
    if (s->N % VFULL == 0 && s->P % VFULL == 0 && aligned16(U) && aligned16(B) && aligned16(C) && aligned16(pp.b_scale) &&
        aligned16(pp.c_scale)) {
      const long long bits = (long long)(reinterpret_cast<uintptr_t>(value) | reinterpret_cast<uintptr_t>(bc)) |
                             s->value_stride * (long long)sizeof(T_) | s->bc_stride * (long long)sizeof(T_);
      al = bits % 16 == 0 ? 16 : bits % 8 == 0 ? 8 : 0;
    }
    // the rows of the any-width kernel, and the scales that it reads in the same vectors
    const int vec = aligned16(pp.b_scale) && aligned16(pp.c_scale) ? pick_vec<T_>(s, {value, bc, U, B, C}) : 1;
    if (al && G) {
      rc = al == 16 ? launch_prep_fwd_lanes<T_, 16>(G, s, d, value, params, bc, pp, U, M, K, B, C, st)
                    : launch_prep_fwd_lanes<T_, 8>(G, s, d, value, params, bc, pp, U, M, K, B, C, st);
    } else if (vec == VFULL) {
      rc = launch_prep_fwd_any<T_, VFULL>(s, d, value, params, bc, pp, U, M, K, B, C, st);
    } else if (vec == VFULL / 2) {
      rc = launch_prep_fwd_any<T_, VFULL / 2>(s, d, value, params, bc, pp, U, M, K, B, C, st);
    } else {
      rc = launch_prep_fwd_any<T_, 1>(s, d, value, params, bc, pp, U, M, K, B, C, st);
    }
  });
  return rc;
}

static int prep_bwd_impl(const slx_prep_shape *s, const void *params, const void *bc, const PrepParams &pp,
                         const void *dU, const float *dM, const float *dK, const void *dB, const void *dC,
                         void *d_value, void *d_params, void *d_bc, const PrepParamGrads &pg, void *workspace,
                         size_t workspace_bytes, void *stream) {
  PrepDims d;
  int rc = check_prep(s, &d);
  if (rc) return rc;
  SLX_REQUIRE(params && bc && dU && dM && dK && dB && dC && d_value && d_params && d_bc, SLX_E_NULL,
              "scanprep_bwd: NULL tensor");
  d.wide_params = params_rows_wide(s, params);
  size_t need = slx_scanprep_bwd_workspace_bytes(s);
  SLX_REQUIRE(workspace && workspace_bytes >= need, SLX_E_WORKSPACE, "scanprep_bwd: workspace of %zu bytes needed",
              need);
  cudaStream_t st = as_stream(stream);
  float *part = static_cast<float *>(workspace);
  SLX_PREP_T(s->dtype, {
    int vec = pick_vec<T_>(s, {bc, dU, dB, dC, d_value, d_bc});
    constexpr int VFULL = 16 / (int)sizeof(T_);
    const int G = prep_lanes<T_>(s);
    const long long bits = (long long)reinterpret_cast<uintptr_t>(bc) | s->bc_stride * (long long)sizeof(T_);
    const bool rows_ok = s->N % VFULL == 0 && s->P % VFULL == 0 && aligned16(dU) && aligned16(dB) && aligned16(dC) &&
                         aligned16(d_value) && aligned16(d_bc) && aligned16(pp.b_scale) && aligned16(pp.c_scale);
    if (G && rows_ok && bits % 16 == 0)
      rc = launch_prep_bwd_lanes<T_, 16>(G, s, d, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, part,
                                         st);
    else if (G && rows_ok && bits % 8 == 0)
      rc = launch_prep_bwd_lanes<T_, 8>(G, s, d, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, part,
                                        st);
    else if (vec == VFULL)
      rc = launch_prep_bwd<T_, VFULL>(s, d, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, part, st);
    else if (vec == VFULL / 2)
      rc = launch_prep_bwd<T_, VFULL / 2>(s, d, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, part,
                                          st);
    else rc = launch_prep_bwd<T_, 1>(s, d, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, part, st);
  });
  return rc;
}

extern "C" {

int slx_scanprep_fwd(const slx_prep_shape *s, const void *value, const void *params, const void *bc,
                     const float *bias, const float *scale, void *U, float *M, float *K, void *B, void *C,
                     void *stream) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  SLX_REQUIRE(bias != nullptr, SLX_E_NULL, "scanprep_fwd: NULL tensor");
  SLX_REQUIRE(!s->normalize_bc || scale, SLX_E_NULL, "scanprep_fwd: scale is NULL with normalize_bc set");
  return prep_fwd_impl(s, value, params, bc, f32_prep_params(s, bias, scale), U, M, K, B, C, stream);
}

int slx_scanprep_fwd_params(const slx_prep_shape *s, const void *value, const void *params, const void *bc,
                            const slx_prep_params *p, void *U, float *M, float *K, void *B, void *C, void *stream) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  PrepParams pp;
  int rc = make_prep_params(s, p, &pp);
  if (rc) return rc;
  return prep_fwd_impl(s, value, params, bc, pp, U, M, K, B, C, stream);
}

size_t slx_scanprep_bwd_workspace_bytes(const slx_prep_shape *s) {
  PrepDims d;
  if (check_prep(s, &d)) return 0;
  // the scalar mapping needs the most tiles-independent space; both use the same tile count
  return prep_bwd_plan(s, 1).ws_bytes;
}

int slx_scanprep_bwd(const slx_prep_shape *s, const void *params, const void *bc, const float *bias,
                     const float *scale, const void *dU, const float *dM, const float *dK, const void *dB,
                     const void *dC, void *d_value, void *d_params, void *d_bc, float *d_bias, float *d_scale,
                     void *workspace, size_t workspace_bytes, void *stream) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  SLX_REQUIRE(bias && d_bias, SLX_E_NULL, "scanprep_bwd: NULL tensor");
  SLX_REQUIRE(!s->normalize_bc || (scale && d_scale), SLX_E_NULL, "scanprep_bwd: scale/d_scale NULL");
  PrepParamGrads pg{};
  pg.bias13 = d_bias;
  pg.b_scale = d_scale;
  pg.c_scale = d_scale ? d_scale + 2 * s->N : nullptr;
  pg.dtype = SLX_F32;
  pg.scale_stride = 4LL * s->N;
  return prep_bwd_impl(s, params, bc, f32_prep_params(s, bias, scale), dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg,
                       workspace, workspace_bytes, stream);
}

int slx_scanprep_bwd_params(const slx_prep_shape *s, const void *params, const void *bc, const slx_prep_params *p,
                            const void *dU, const float *dM, const float *dK, const void *dB, const void *dC,
                            void *d_value, void *d_params, void *d_bc, void *d_bias, void *d_b_scale, void *d_c_scale,
                            void *workspace, size_t workspace_bytes, void *stream) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "shape is NULL");
  PrepParams pp;
  int rc = make_prep_params(s, p, &pp);
  if (rc) return rc;
  SLX_REQUIRE(d_bias && (!s->normalize_bc || (d_b_scale && d_c_scale)), SLX_E_NULL, "scanprep_bwd: NULL gradient");
  PrepParamGrads pg{};
  const size_t row = (size_t)s->heads * (p->dtype == SLX_F32 ? 4 : 2);
  for (int k = 0; k < 7; ++k) pg.bias[k] = static_cast<char *>(d_bias) + k * row;
  pg.b_scale = d_b_scale;
  pg.c_scale = d_c_scale;
  pg.dtype = p->dtype;
  pg.scale_stride = 2LL * s->N;
  return prep_bwd_impl(s, params, bc, pp, dU, dM, dK, dB, dC, d_value, d_params, d_bc, pg, workspace, workspace_bytes,
                       stream);
}

}  // extern "C"
