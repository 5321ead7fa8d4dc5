// fp32-exact chunk kernels of the v2x2ssd scan (CUDA-core FFMA path).
//
// One CTA of 256 threads per (chunk, batch*head).  All contractions are done
// with fp32 FMAs on shared-memory tiles, so that fp32 inputs reproduce the
// reference to ~1e-6; half inputs are widened on load.
//
// Math (per chunk, local token index t, s in [0,L)):
//   p_t   = prod_{tau<=t} m_tau = exp(lp_t) * phi_t            (stable split)
//   gamma_s = m_{s+1} k^c_s + k^p_{s+1}                         (merged taps)
//   h_t = p_t z0 + (p_t/p_0) k^p_0 x_{-1} + sum_{s<t} (p_t/p_{s+1}) gamma_s x_s
//         + k^c_t x_t ,    x_s = u_s (x) b_s ,   y_t = Re <c_t, h_t>
// which is the reference recurrence (slinoss/ops/v2x2ssd/reference.py:704-803)
// with the two taps of source token s folded into one coefficient.
// With Qbar_t = c_t conj(phi_t) and kappa_s = gamma_s b_s conj(phi_{s+1}) stored
// as interleaved (re,im) floats, Re(conj(c_t) (p_t/p_{s+1}) gamma_s b_s) is the
// plain real dot <Qbar_t, kappa_s> times exp(lp_t - lp_{s+1}).
#pragma once

#include "common.cuh"

namespace slx {

__device__ int g_scan_bad = 0;  // becomes 1 when a kernel met a transition of magnitude exactly 0

constexpr int kThreads = 256;
constexpr int kPMax = 64;

struct ScanDims {
  int BH, T, P, N, D, L, NC;
};

template <typename T>
__device__ __forceinline__ float2 load_pair(const T *p);
template <>
__device__ __forceinline__ float2 load_pair<float>(const float *p) {
  return *reinterpret_cast<const float2 *>(p);
}
template <>
__device__ __forceinline__ float2 load_pair<__nv_bfloat16>(const __nv_bfloat16 *p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p));
}
template <>
__device__ __forceinline__ float2 load_pair<__half>(const __half *p) {
  return __half22float2(*reinterpret_cast<const __half2 *>(p));
}
// The streaming row of batch-head offset `off` when it is held in the activation dtype (the same loads as any other
// row then), NULL when it is absent or fp32.
template <typename T>
__device__ __forceinline__ const T *prev_row(const void *p, int dtype, size_t off) {
  return (p != nullptr && dtype != SLX_F32) ? static_cast<const T *>(p) + off : nullptr;
}
template <typename T>
__device__ __forceinline__ void store_pair(T *p, float2 v);
template <>
__device__ __forceinline__ void store_pair<float>(float *p, float2 v) {
  *reinterpret_cast<float2 *>(p) = v;
}
template <>
__device__ __forceinline__ void store_pair<__nv_bfloat16>(__nv_bfloat16 *p, float2 v) {
  *reinterpret_cast<__nv_bfloat162 *>(p) = __float22bfloat162_rn(v);
}
template <>
__device__ __forceinline__ void store_pair<__half>(__half *p, float2 v) {
  *reinterpret_cast<__half2 *>(p) = __float22half2_rn(v);
}

// sum a float2 over groups of NL consecutive lanes (NL power of two <= 32)
template <int NL>
__device__ __forceinline__ float2 group_sum(float2 v) {
#pragma unroll
  for (int off = NL / 2; off > 0; off >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
  }
  return v;
}

// ---- geometry -----------------------------------------------------------------------------------------------
// 256 threads as 16 (ty) x 16 (tx).  An accumulator tile of L rows gives thread (ty, tx) TM = L/16 rows in groups of
// VM adjacent ones, so that an operand that lies row-adjacent is read as one vector; a warp's rows are adjacent too,
// which lets the products of the causal triangle skip what is masked for all of them.  Head-dim tiles are 16*TP wide
// (TP = 2 for P <= 32, else 4), a thread owns columns TP*tx .. TP*tx+TP-1.  The state is walked in slabs of 32 values;
// a thread owns the complex lane tx of the slab.
// The products are bound by shared-memory wavefronts as soon as operands are read one float at a time (8 loads per 16
// fmas and thread; this was half of the exact kernels' time): every operand is read in vectors along the axis it is
// contiguous in, rows are padded to 4 mod 32 words so that the vectors of 8 rows fill the banks.  What is left is half
// fmas, a third vector loads, the rest staging; two CTAs per SM cover each other's global loads.
// Batch 2, 8 heads, 2048 tokens, P 64, D 128, fp32 (512 chunks of 64): forward 85 -> 53 us, backward 276 -> 148 us,
// increment 33 -> 29 us, dZ0 30 -> 22 us; three CTAs of 32 tokens per SM spilled and were slower (199 us backward).
template <int L>
struct ChunkRows {
  static constexpr int TM = L / 16;
  static constexpr int VM = TM < 4 ? TM : 4;
  __device__ static __forceinline__ int row(int ty, int i) { return VM * ty + (i % VM) + 16 * VM * (i / VM); }
  __device__ static __forceinline__ int warp_min() { return 2 * VM * (threadIdx.x >> 5); }
  __device__ static __forceinline__ int warp_max() { return warp_min() + 2 * VM - 1 + (TM > VM ? 16 * VM * (TM / VM - 1) : 0); }
};
constexpr int kDS = 32;          // state values per slab
constexpr int kLdD = kDS + 4;    // row stride of the slab tiles
template <int TP>
constexpr int ld_p() { return 16 * TP + 4; }
template <int L>
constexpr int ld_l() { return L + 4; }
// slot of head-dim row p in the Z0 / Lambda tiles: thread tx reads its TP rows at tx, tx+16, ... (conflict-free)
template <int TP>
__device__ __forceinline__ int prow(int p) { return (p % TP) * 16 + p / TP; }

// the same of row p + e, for p a multiple of 4 and a compile-time e < 4
template <int TP>
__device__ __forceinline__ int prow4(int p, int e) { return (e % TP) * 16 + p / TP + e / TP; }

template <int N>
__device__ __forceinline__ void ld_vec(const float *p, float (&v)[N]) {
  if constexpr (N == 4) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else if constexpr (N == 2) {
    const float2 q = *reinterpret_cast<const float2 *>(p);
    v[0] = q.x; v[1] = q.y;
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = p[i];
  }
}

// acc[i][j] += sum_k a_i[k] b_j[k], both contiguous in k;  k in [0, k1), multiples of 4
template <int TM, int TN, int TNA, typename FA, typename FB>
__device__ __forceinline__ void mm_kk(float (&acc)[TM][TNA], int k1, FA a, FB b) {
#pragma unroll 2
  for (int k = 0; k < k1; k += 4) {
    float av[TM][4], bv[TN][4];
#pragma unroll
    for (int i = 0; i < TM; ++i) ld_vec<4>(a(i) + k, av[i]);
#pragma unroll
    for (int j = 0; j < TN; ++j) ld_vec<4>(b(j) + k, bv[j]);
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i][e], bv[j][e], acc[i][j]);
  }
}
// the same on the first jn (of TM) 16-column blocks only: the blocks a causal tile needs for this warp's rows
template <int TM, int JN = TM, typename FA, typename FB>
__device__ __forceinline__ void mm_kk_causal(float (&acc)[TM][TM], int jn, int k1, FA a, FB b) {
  if constexpr (JN > 1) {
    if (jn < JN) {
      mm_kk_causal<TM, JN - 1>(acc, jn, k1, a, b);
      return;
    }
  }
  mm_kk<TM, JN>(acc, k1, a, b);
}
// acc[i][j] += sum_k a_i[k] b_k[j]: a contiguous in k, b in the columns, b(k, e) the row k + e < k + 4;  k in [k0, k1),
// multiples of 4
template <int TM, int TN, typename FA, typename FB>
__device__ __forceinline__ void mm_kn(float (&acc)[TM][TN], int k0, int k1, FA a, FB b) {
#pragma unroll 2
  for (int k = k0; k < k1; k += 4) {
    float av[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i) ld_vec<4>(a(i) + k, av[i]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float bv[TN];
      ld_vec<TN>(b(k, e), bv);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i][e], bv[j], acc[i][j]);
    }
  }
}
// acc[i][j] += sum_k a(k)[row_i] b(k)[j]: a contiguous in the rows (a(k) points at the thread's first row)
template <int L, int TN, typename FA, typename FB>
__device__ __forceinline__ void mm_mn(float (&acc)[L / 16][TN], int k0, int k1, FA a, FB b) {
  constexpr int TM = ChunkRows<L>::TM, VM = ChunkRows<L>::VM;
#pragma unroll 4
  for (int k = k0; k < k1; ++k) {
    float av[TM], bv[TN];
#pragma unroll
    for (int g = 0; g < TM / VM; ++g) {
      float t[VM];
      ld_vec<VM>(a(k) + 16 * VM * g, t);
#pragma unroll
      for (int i = 0; i < VM; ++i) av[VM * g + i] = t[i];
    }
    ld_vec<TN>(b(k), bv);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
}

// (L x 16*TP) tile of a (tokens, P) matrix, zero past `valid` tokens and P columns
template <typename T, int L, int TP>
__device__ __forceinline__ void load_head_tile(float *dst, const T *src, int valid, int P) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float v[L / 16][TP];  // all loads first: they may not be moved over the stores
#pragma unroll
  for (int i = 0; i < L / 16; ++i) {
    const int r = ty + 16 * i;
#pragma unroll
    for (int e = 0; e < TP; ++e) v[i][e] = 0.f;
    if (r >= valid) continue;
    const T *p = src + (size_t)r * P + TP * tx;
    if (P == 16 * TP) {
#pragma unroll
      for (int e = 0; e < TP; e += 2) {
        const float2 q = load_pair<T>(p + e);
        v[i][e] = q.x;
        v[i][e + 1] = q.y;
      }
    } else {
#pragma unroll
      for (int e = 0; e < TP; ++e)
        if (TP * tx + e < P) v[i][e] = to_f(p[e]);
    }
  }
#pragma unroll
  for (int i = 0; i < L / 16; ++i) {
    float *o = dst + (ty + 16 * i) * ld_p<TP>() + TP * tx;
#pragma unroll
    for (int e = 0; e < TP; e += 2) *reinterpret_cast<float2 *>(o + e) = make_float2(v[i][e], v[i][e + 1]);
  }
}
// TP adjacent head-dim values of one token
template <typename T, int TP>
__device__ __forceinline__ void store_head(T *p, int col, int P, const float (&v)[TP]) {
  if (P == 16 * TP) {
#pragma unroll
    for (int e = 0; e < TP; e += 2) store_pair<T>(p + col + e, make_float2(v[e], v[e + 1]));
  } else {
#pragma unroll
    for (int e = 0; e < TP; ++e)
      if (col + e < P) p[col + e] = from_f<T>(v[e]);
  }
}
// (P x 32) slab of a chunk state, row p in slot prow(p): this thread's TP rows of complex lane dd/2, and their store
template <int TP>
__device__ __forceinline__ void load_state_slab(float2 (&v)[TP], const float *src, int P, int D, int dd) {
#pragma unroll
  for (int j = 0; j < TP; ++j) {
    const int p = TP * (threadIdx.x >> 4) + j;
    v[j] = p < P && dd < D ? *reinterpret_cast<const float2 *>(src + (size_t)p * D + dd) : make_float2(0.f, 0.f);
  }
}
template <int TP>
__device__ __forceinline__ void store_state_slab(float *dst, const float2 (&v)[TP]) {
#pragma unroll
  for (int j = 0; j < TP; ++j)
    *reinterpret_cast<float2 *>(dst + (16 * j + (threadIdx.x >> 4)) * kLdD + 2 * (threadIdx.x & 15)) = v[j];
}
// complex lane dd/2 of the chunk's rows ty + 16 i of C and B, zero past `valid` and D
template <typename T, int L>
__device__ __forceinline__ void load_cb(float2 (&cv)[L / 16], float2 (&bv)[L / 16], const T *C, const T *B, int valid,
                                        int D, int dd) {
#pragma unroll
  for (int i = 0; i < L / 16; ++i) {
    const int r = (threadIdx.x >> 4) + 16 * i;
    cv[i] = bv[i] = make_float2(0.f, 0.f);
    if (r < valid && dd < D) {
      cv[i] = load_pair<T>(C + (size_t)r * D + dd);
      bv[i] = load_pair<T>(B + (size_t)r * D + dd);
    }
  }
}
// complex lane dd/2 of the token in front of the chunk
template <typename T, typename Args>
__device__ __forceinline__ float2 prev_b(const T *B, const Args &a, int t0, size_t tok0, int bh, int dd) {
  if (dd >= a.d.D) return make_float2(0.f, 0.f);
  if (t0 > 0) return load_pair<T>(B + (tok0 - 1) * a.d.D + dd);
  if (a.Bprev) return load_as_f2(a.Bprev, a.prev_dtype, (size_t)bh * a.d.D + dd);
  return make_float2(0.f, 0.f);
}
template <typename T, typename Args>
__device__ __forceinline__ float prev_u(const T *U, const Args &a, int t0, size_t tok0, int bh, int p) {
  if (p >= a.d.P) return 0.f;
  if (t0 > 0) return to_f(U[(tok0 - 1) * a.d.P + p]);
  if (a.Uprev) return load_as_f(a.Uprev, a.prev_dtype, (size_t)bh * a.d.P + p);
  return 0.f;
}
__device__ __forceinline__ void load_taps_rows(const float *K, size_t tok0, int L, int valid, float2 *kp, float2 *kc) {
  for (int t = threadIdx.x; t < L; t += kThreads) {
    float2 vp = make_float2(0.f, 0.f), vc = vp;
    if (t < valid) {
      const float4 k4 = *reinterpret_cast<const float4 *>(K + (tok0 + t) * 4);
      vp = make_float2(k4.x, k4.y);
      vc = make_float2(k4.z, k4.w);
    }
    kp[t] = vp;
    kc[t] = vc;
  }
}

// ---------------------------------------------------------------------------
// out[p, :] = sum_t A[t, p] * (coef_t * x_t[:])  (+ rank-1 boundary term)
// MODE 0: chunk increment.  A = U, x = B, coef_s = sigma_{s+1} gamma_s (= the
//         weight of source token s in the chunk-final state); boundary
//         u_{-1} (x) sigma_0 k^p_0 b_{-1}; also writes m_chunk.
//         Replaces reference.py:937 (chunk_increment).
// MODE 1: dZ0.  A = dY, x = C, coef_t = conj(p_t).
template <typename T>
struct OuterArgs {
  const T *A;       // (BH,T,P)
  const T *X;       // (BH,T,D)
  const float *M;   // (BH,T,2)
  const float *K;   // (BH,T,2,2)  (mode 0)
  const void *Bprev, *Uprev;  // (BH,D), (BH,P), nullable (mode 0)
  int prev_dtype;
  float *out;       // (BH,NC,P,D)
  float *m_chunk;   // (BH,NC,2) (mode 0)
  ScanDims d;
};
constexpr int kOuterDS = 64;
template <int L, int TP>
constexpr size_t outer_smem_bytes() {
  return sizeof(float) * (size_t)(L * ld_p<TP>() + L * (kOuterDS + 4) + L + 2 * L * 3 + 16 * TP);
}

template <typename T, int L, int TP, int MODE>
__global__ void __launch_bounds__(kThreads) chunk_outer_kernel(OuterArgs<T> a) {
  constexpr int LP = ld_p<TP>(), LX = kOuterDS + 4;
  extern __shared__ __align__(16) float sm[];
  float *As = sm;              // [L][LP]
  float *Xs = As + L * LP;     // [L][LX]
  float *lp = Xs + L * LX;
  float2 *ph = reinterpret_cast<float2 *>(lp + L), *mraw = ph + L, *coef = mraw + L;
  float *um1 = reinterpret_cast<float *>(coef + L);

  const ScanDims d = a.d;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int t0 = c * L;
  const int valid = min(L, d.T - t0);
  const size_t tok0 = (size_t)bh * d.T + t0;

  chunk_prefix_warp0(a.M + tok0 * 2, L, valid, lp, ph, mraw, &g_scan_bad);
  load_head_tile<T, L, TP>(As, a.A + tok0 * d.P, valid, d.P);
  if (MODE == 0 && tid < 16 * TP) um1[tid] = prev_u<T>(a.A, a, t0, tok0, bh, tid);
  __syncthreads();
  // per-row coefficient
  float2 k0p = make_float2(0.f, 0.f);
  for (int t = tid; t < L; t += kThreads) {
    float2 cf;
    if (MODE == 0) {
      float2 kc = make_float2(0.f, 0.f), kpn = make_float2(0.f, 0.f);
      if (t < valid) kc = *reinterpret_cast<const float2 *>(a.K + (tok0 + t) * 4 + 2);
      if (t + 1 < valid) kpn = *reinterpret_cast<const float2 *>(a.K + (tok0 + t + 1) * 4);
      if (t + 1 < L) {
        float2 gam = cadd(cmul(mraw[t + 1], kc), kpn);
        float2 sig = cscale(cmulc(ph[L - 1], ph[t + 1]), expf(lp[L - 1] - lp[t + 1]));
        cf = cmul(sig, gam);
      } else {
        cf = kc;
      }
    } else {
      cf = cscale(cconj(ph[t]), expf(lp[t]));
    }
    coef[t] = cf;
  }
  if (MODE == 0 && tid >= kThreads - 32) {
    // chunk transition by direct product (reference.py:509-516 accumulates the same product in its reverse scan):
    // adjacent tokens per lane, then a butterfly in token order
    const int lane = tid & 31;
    float2 acc = make_float2(1.f, 0.f);
#pragma unroll
    for (int i = 0; i < (L + 31) / 32; ++i) {
      const int t = lane * ((L + 31) / 32) + i;
      if (t < L) acc = cmul(acc, mraw[t]);
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float ox = __shfl_xor_sync(0xffffffffu, acc.x, off), oy = __shfl_xor_sync(0xffffffffu, acc.y, off);
      acc = cmul(acc, make_float2(ox, oy));
    }
    if (lane == 0) *reinterpret_cast<float2 *>(a.m_chunk + ((size_t)bh * d.NC + c) * 2) = acc;
  }
  if (MODE == 0) {  // weight of the boundary source: (p_{L-1}/p_0) k^p_0
    k0p = *reinterpret_cast<const float2 *>(a.K + tok0 * 4);
    k0p = cmul(cscale(cmulc(ph[L - 1], ph[0]), expf(lp[L - 1] - lp[0])), k0p);
  }
  __syncthreads();

  float *outc = a.out + ((size_t)bh * d.NC + c) * d.P * d.D;
  for (int d0 = 0; d0 < d.D; d0 += kOuterDS) {
    const int dd = d0 + 4 * tx;
    float2 x0[L / 16], x1[L / 16];
#pragma unroll
    for (int i = 0; i < L / 16; ++i) {
      const int r = ty + 16 * i;
      x0[i] = x1[i] = make_float2(0.f, 0.f);
      if (r < valid) {
        if (dd < d.D) x0[i] = load_pair<T>(a.X + (tok0 + r) * d.D + dd);
        if (dd + 2 < d.D) x1[i] = load_pair<T>(a.X + (tok0 + r) * d.D + dd + 2);
      }
    }
#pragma unroll
    for (int i = 0; i < L / 16; ++i) {
      const int r = ty + 16 * i;
      const float2 c0 = cmul(coef[r], x0[i]), c1 = cmul(coef[r], x1[i]);
      *reinterpret_cast<float4 *>(Xs + r * LX + 4 * tx) = make_float4(c0.x, c0.y, c1.x, c1.y);
    }
    __syncthreads();
    float acc[TP][4];  // rows TP*ty + i, columns 4 tx + j
#pragma unroll
    for (int i = 0; i < TP; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    mm_mn<16 * TP, 4>(acc, 0, L, [&](int k) { return As + k * LP + TP * ty; },
                      [&](int k) { return Xs + k * LX + 4 * tx; });
    float2 b0 = make_float2(0.f, 0.f), b1 = b0;
    if (MODE == 0) {
      b0 = cmul(k0p, prev_b<T>(a.X, a, t0, tok0, bh, dd));
      b1 = cmul(k0p, prev_b<T>(a.X, a, t0, tok0, bh, dd + 2));
    }
#pragma unroll
    for (int i = 0; i < TP; ++i) {
      const int p = TP * ty + i;
      if (p >= d.P) continue;
      const float u = MODE == 0 ? um1[p] : 0.f;
      float *o = outc + (size_t)p * d.D + dd;
      if (dd < d.D) *reinterpret_cast<float2 *>(o) = make_float2(fmaf(u, b0.x, acc[i][0]), fmaf(u, b0.y, acc[i][1]));
      if (dd + 2 < d.D)
        *reinterpret_cast<float2 *>(o + 2) = make_float2(fmaf(u, b1.x, acc[i][2]), fmaf(u, b1.y, acc[i][3]));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Forward chunk scan.  Replaces reference.py:1059 (chunk_scan).
template <typename T>
struct ScanFwdArgs {
  const T *U, *B, *C;
  const float *M, *K, *starts;
  const void *Bprev, *Uprev;
  int prev_dtype;
  T *Y;
  int *bad;  // unused (the kernels report through g_scan_bad)
  ScanDims d;
};
template <int L, int TP>
constexpr size_t scan_fwd_smem_bytes() {
  return sizeof(float) * (size_t)(L * ld_p<TP>() + 2 * L * kLdD + 16 * TP * kLdD + L * ld_l<L>() + 2 * L + 2 * L * 6 + 16 * TP);
}

template <typename T, int L, int TP>
__global__ void __launch_bounds__(kThreads, L <= 64 ? 2 : 1) chunk_scan_fwd_kernel(ScanFwdArgs<T> a) {
  using R = ChunkRows<L>;
  constexpr int TM = R::TM, LP = ld_p<TP>(), LL = ld_l<L>();
  extern __shared__ __align__(16) float sm[];
  float *Us = sm;                     // [L][LP]
  float *Qs = Us + L * LP;            // [L][36]
  float *Ks = Qs + L * kLdD;          // [L][36]
  float *Zs = Ks + L * kLdD;          // [16 TP][36]
  float *Ss = Zs + 16 * TP * kLdD;    // [L][LL]
  float *lp = Ss + L * LL, *sg = lp + L;
  float2 *ph = reinterpret_cast<float2 *>(sg + L);
  float2 *mraw = ph + L, *kc = mraw + L, *kp = kc + L, *gk = kp + L, *cb = gk + L;
  float *um1 = reinterpret_cast<float *>(cb + L);

  const ScanDims d = a.d;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int t0 = c * L;
  const int valid = min(L, d.T - t0);
  const size_t tok0 = (size_t)bh * d.T + t0;

  chunk_prefix_warp0(a.M + tok0 * 2, L, valid, lp, ph, mraw, &g_scan_bad);
  load_taps_rows(a.K, tok0, L, valid, kp, kc);
  load_head_tile<T, L, TP>(Us, a.U + tok0 * d.P, valid, d.P);
  if (tid < 16 * TP) um1[tid] = prev_u<T>(a.U, a, t0, tok0, bh, tid);
  __syncthreads();
  for (int t = tid; t < L; t += kThreads)  // gamma_t conj(phi_{t+1})
    gk[t] = t + 1 < L ? cmulc(cadd(cmul(mraw[t + 1], kc[t]), kp[t + 1]), ph[t + 1]) : make_float2(0.f, 0.f);
  __syncthreads();

  float S[TM][TM], Yo[TM][TP];
  float2 acc_cb[TM];  // conj(c) b of rows ty + 16 i
  float acc_s[TM];    // boundary score of the same rows
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < TM; ++j) S[i][j] = 0.f;
#pragma unroll
    for (int j = 0; j < TP; ++j) Yo[i][j] = 0.f;
    acc_cb[i] = make_float2(0.f, 0.f);
    acc_s[i] = 0.f;
  }
  const float *z0 = a.starts + ((size_t)bh * d.NC + c) * d.P * d.D;
  const int jn = R::warp_max() / 16 + 1;

  for (int d0 = 0; d0 < d.D; d0 += kDS) {
    const int dd = d0 + 2 * tx;
    // every load of the slab before the first store, which no load may be moved over
    float2 cv[TM], bv[TM], zv[TP];
    load_cb<T, L>(cv, bv, a.C + tok0 * d.D, a.B + tok0 * d.D, valid, d.D, dd);
    load_state_slab<TP>(zv, z0, d.P, d.D, dd);
    const float2 km = cmul(cmulc(kp[0], ph[0]), prev_b<T>(a.B, a, t0, tok0, bh, dd));  // k^p_0 conj(phi_0) b_{-1}
    store_state_slab<TP>(Zs, zv);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int r = ty + 16 * i;
      const float2 q = cmulc(cv[i], ph[r]);
      *reinterpret_cast<float2 *>(Qs + r * kLdD + 2 * tx) = q;
      *reinterpret_cast<float2 *>(Ks + r * kLdD + 2 * tx) = cmul(gk[r], bv[i]);
      acc_cb[i] = cadd(acc_cb[i], cmul(cconj(cv[i]), bv[i]));
      acc_s[i] = fmaf(q.x, km.x, fmaf(q.y, km.y, acc_s[i]));
    }
    __syncthreads();
    auto qrow = [&](int i) { return Qs + R::row(ty, i) * kLdD; };
    mm_kk_causal<TM>(S, jn, kDS, qrow, [&](int j) { return Ks + (tx + 16 * j) * kLdD; });
    mm_kk<TM, TP>(Yo, kDS, qrow, [&](int j) { return Zs + (tx + 16 * j) * kLdD; });
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = ty + 16 * i;
    const float2 s = group_sum<16>(acc_cb[i]), w = group_sum<16>(make_float2(acc_s[i], 0.f));
    if (tx == 0) {
      cb[r] = s;
      sg[r] = expf(lp[r] - lp[0]) * w.x;  // weight of the token in front of the chunk
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int t = R::row(ty, i);
    const float el = expf(lp[t]);
#pragma unroll
    for (int j = 0; j < TP; ++j) Yo[i][j] *= el;
#pragma unroll
    for (int j = 0; j < TM; ++j) {
      const int s = tx + 16 * j;
      float v = 0.f;
      if (s < t) v = S[i][j] * expf(lp[t] - lp[s + 1]);
      else if (s == t) v = kc[t].x * cb[t].x - kc[t].y * cb[t].y;
      Ss[t * LL + s] = v;
    }
  }
  __syncthreads();
  mm_kn<TM, TP>(Yo, 0, (R::warp_max() + 4) & ~3, [&](int i) { return Ss + R::row(ty, i) * LL; },
                [&](int k, int e) { return Us + (k + e) * LP + TP * tx; });
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int t = R::row(ty, i);
    if (t >= valid) continue;
    float y[TP];
#pragma unroll
    for (int j = 0; j < TP; ++j) y[j] = fmaf(sg[t], um1[TP * tx + j], Yo[i][j]);
    store_head<T, TP>(a.Y + (tok0 + t) * d.P, TP * tx, d.P, y);
  }
}

// ---------------------------------------------------------------------------
// Backward of one chunk, given d_inc[c] = dL/d(chunk-final state) and the
// chunk's start state.  Writes dU, dB, dC (activation dtype), dM, dK (fp32) for
// the chunk's tokens, and the gradient carried to the token before the chunk
// (carryB (BH,NC,D), carryU (BH,NC,P)), which a follow-up kernel adds to the
// previous chunk's last row (or returns as dB_prev/dU_prev for chunk 0).
//
// With Lambda' = conj(phi_{L-1}) Lambda, es_s = exp(lp_{L-1} - lp_{s+1}) (1 for the last row), psi_s = phi_{s+1}
// (phi_{L-1} for the last row) and kappa_s = gamma_s conj(psi_s) b_s (gamma_{L-1} = k^c_{L-1}), both paths of a
// source token share one accumulator:
//   X_s = sum_t dS'[t][s] Qbar_t + es_s u_s . Lambda',    dB_s = conj(k^c_s) G_ss c_s + conj(gamma_s) psi_s X_s
//   dU_s = sum_t S'[t][s] dY_t + es_s <kappa_s, Lambda'>
// The token in front of the chunk is a rank-one term of dq, a column sum of X's kind and two dots.
//
// dM uses the identity (local prefix p_tau; all quantities per chunk)
//   conj(p_tau) dL/dp_tau = sum_n c_tau conj(dC_tau) - conj(k^c_tau) dk^c_tau
//                           - conj(k^p_tau) dk^p_tau + [tau = L-1] <z_end, d_inc>
//   dM_t = (sum_{tau >= t} conj(p_tau) dL/dp_tau) / conj(m_t)
// so no per-token state is ever materialised.
template <typename T>
struct ScanBwdArgs {
  const T *U, *B, *C, *dY;
  const float *M, *K, *starts, *d_inc, *zdot;
  const void *Bprev, *Uprev;
  int prev_dtype;
  T *dU, *dB, *dC;
  float *dM, *dK, *carryB, *carryU;
  ScanDims d;
};
template <int L, int TP>
constexpr size_t scan_bwd_smem_bytes() {
  return sizeof(float) * (size_t)(2 * L * ld_p<TP>() + L * ld_l<L>() + 2 * L * kLdD + 2 * 16 * TP * kLdD + 16 * kDS +
                                  4 * L + 2 * L * 9 + 2 * 16 * TP + kDS + 8);
}

template <typename T, int L, int TP>
__global__ void __launch_bounds__(kThreads, L <= 64 ? 2 : 1) chunk_scan_bwd_kernel(ScanBwdArgs<T> a) {
  using R = ChunkRows<L>;
  constexpr int TM = R::TM, LP = ld_p<TP>(), LL = ld_l<L>();
  extern __shared__ __align__(16) float sm[];
  float *dYs = sm;                    // [L][LP]
  float *Us = dYs + L * LP;           // [L][LP]
  float *dSs = Us + L * LP;           // [L][LL]  dS', at the end S'
  float *Qs = dSs + L * LL;           // [L][36]  Qbar
  float *Ks = Qs + L * kLdD;          // [L][36]  kappa
  float *Zs = Ks + L * kLdD;          // [16 TP][36]  Z0 (rows by prow)
  float *Ls = Zs + 16 * TP * kLdD;    // [16 TP][36]  Lambda'
  float *red = Ls + 16 * TP * kLdD;   // [16][32]  partials of the carried gradient
  float *lp = red + 16 * kDS, *gd = lp + L, *wv = gd + L, *sg = wv + L;
  float2 *ph = reinterpret_cast<float2 *>(sg + L);
  float2 *mraw = ph + L, *kc = mraw + L, *kp = kc + L, *gk = kp + L, *bc = gk + L, *bX = bc + L, *gA = bX + L,
         *gsum = gA + L;
  float *um1 = reinterpret_cast<float *>(gsum + L);
  float *duc = um1 + 16 * TP;
  float *km1 = duc + 16 * TP;                                // [32] kappa_{-1} of the slab
  float2 *misc = reinterpret_cast<float2 *>(km1 + kDS);      // [0] dk^p_0

  const ScanDims d = a.d;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int t0 = c * L;
  const int valid = min(L, d.T - t0);
  const size_t tok0 = (size_t)bh * d.T + t0;

  chunk_prefix_warp0(a.M + tok0 * 2, L, valid, lp, ph, mraw, &g_scan_bad);
  load_taps_rows(a.K, tok0, L, valid, kp, kc);
  load_head_tile<T, L, TP>(Us, a.U + tok0 * d.P, valid, d.P);
  load_head_tile<T, L, TP>(dYs, a.dY + tok0 * d.P, valid, d.P);
  if (tid < 16 * TP) um1[tid] = prev_u<T>(a.U, a, t0, tok0, bh, tid);
  __syncthreads();
  for (int t = tid; t < L; t += kThreads)
    gk[t] = t + 1 < L ? cmulc(cadd(cmul(mraw[t + 1], kc[t]), kp[t + 1]), ph[t + 1]) : cmulc(kc[t], ph[t]);
#pragma unroll
  for (int i = 0; i < TM; ++i) {  // w_t = exp(lp_t - lp_0) dY_t . u_{-1}
    const int r = ty + 16 * i;
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < TP; ++e) s = fmaf(dYs[r * LP + TP * tx + e], um1[TP * tx + e], s);
    const float2 g = group_sum<16>(make_float2(s, 0.f));
    if (tx == 0) wv[r] = expf(lp[r] - lp[0]) * g.x;
  }
  const int jn = R::warp_max() / 16 + 1;
  const int p4 = (d.P + 3) & ~3;
  // ---- G = dY U^T, dS' = G * exp(lp_t - lp_{s+1}) on s < t ---------------------
  {
    float G[TM][TM];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TM; ++j) G[i][j] = 0.f;
    mm_kk_causal<TM>(G, jn, p4, [&](int i) { return dYs + R::row(ty, i) * LP; },
                     [&](int j) { return Us + (tx + 16 * j) * LP; });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int t = R::row(ty, i);
#pragma unroll
      for (int j = 0; j < TM; ++j) {
        const int s = tx + 16 * j;
        dSs[t * LL + s] = (s < t) ? G[i][j] * expf(lp[t] - lp[s + 1]) : 0.f;
        if (s == t) gd[t] = G[i][j];
      }
    }
  }
  // per-row factors of this thread's accumulator rows
  float el[TM], es[TM];
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int t = R::row(ty, i);
    el[i] = expf(lp[t]);
    es[i] = t + 1 < L ? expf(lp[L - 1] - lp[t + 1]) : 1.f;
  }
  const float es0 = expf(lp[L - 1] - lp[0]);

  float S[TM][TM], dU[TM][TP];
  float2 acc_bc[TM], pgA[TM], pP[TM];  // acc_bc: rows ty + 16 i; the others: accumulator rows
  float acc_s[TM], acc_du = 0.f;
  float2 dkp0 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < TM; ++j) S[i][j] = 0.f;
#pragma unroll
    for (int j = 0; j < TP; ++j) dU[i][j] = 0.f;
    acc_bc[i] = pgA[i] = pP[i] = make_float2(0.f, 0.f);
    acc_s[i] = 0.f;
  }
  const float *z0 = a.starts + ((size_t)bh * d.NC + c) * d.P * d.D;
  const float *lam = a.d_inc + ((size_t)bh * d.NC + c) * d.P * d.D;
  float *cB = a.carryB + ((size_t)bh * d.NC + c) * d.D;
  __syncthreads();  // dS', gd

  for (int d0 = 0; d0 < d.D; d0 += kDS) {
    const int dd = d0 + 2 * tx;
    const bool on = dd < d.D;
    // ---- stage the slab: every load before the first store, which no load may be moved over ----
    float2 cv[TM], bv[TM], zv[TP], lv[TP];
    load_cb<T, L>(cv, bv, a.C + tok0 * d.D, a.B + tok0 * d.D, valid, d.D, dd);
    load_state_slab<TP>(zv, z0, d.P, d.D, dd);
    load_state_slab<TP>(lv, lam, d.P, d.D, dd);
    const float2 bm = prev_b<T>(a.B, a, t0, tok0, bh, dd);
    const float2 km = cmul(cmulc(kp[0], ph[0]), bm);  // k^p_0 conj(phi_0) b_{-1}
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int r = ty + 16 * i;
      const float2 q = cmulc(cv[i], ph[r]);
      *reinterpret_cast<float2 *>(Qs + r * kLdD + 2 * tx) = q;
      *reinterpret_cast<float2 *>(Ks + r * kLdD + 2 * tx) = cmul(gk[r], bv[i]);
      acc_bc[i] = cadd(acc_bc[i], cmul(cconj(bv[i]), cv[i]));
      acc_s[i] = fmaf(q.x, km.x, fmaf(q.y, km.y, acc_s[i]));
    }
#pragma unroll
    for (int j = 0; j < TP; ++j) lv[j] = cmulc(lv[j], ph[L - 1]);
    store_state_slab<TP>(Zs, zv);
    store_state_slab<TP>(Ls, lv);
    if (ty == 0) *reinterpret_cast<float2 *>(km1 + 2 * tx) = km;
    __syncthreads();

    // ---- scores, increment path of dU --------------------------------------
    mm_kk_causal<TM>(S, jn, kDS, [&](int i) { return Qs + R::row(ty, i) * kLdD; },
                     [&](int j) { return Ks + (tx + 16 * j) * kLdD; });
    mm_kk<TM, TP>(dU, kDS, [&](int i) { return Ks + R::row(ty, i) * kLdD; },
                  [&](int j) { return Ls + (tx + 16 * j) * kLdD; });
    if (tid < 64 * TP) {  // kappa_{-1} . Lambda'[p], a quarter of the slab per thread
      const int p = tid >> 2, k0 = 8 * (tid & 3);
      const float *lr = Ls + prow<TP>(p) * kLdD + k0;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc_du = fmaf(km1[k0 + e], lr[e], acc_du);
    }
    // the gradient of the token in front of the chunk: sum_t w_t Qbar_t + es_{-1} u_{-1} . Lambda', by ty
    {
      float2 x = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < TP; ++j) {
        const float u = es0 * um1[TP * ty + j];
        const float2 l = *reinterpret_cast<const float2 *>(Ls + (16 * j + ty) * kLdD + 2 * tx);
        x.x = fmaf(u, l.x, x.x);
        x.y = fmaf(u, l.y, x.y);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int r = ty + 16 * i;
        const float2 q = *reinterpret_cast<const float2 *>(Qs + r * kLdD + 2 * tx);
        x.x = fmaf(wv[r], q.x, x.x);
        x.y = fmaf(wv[r], q.y, x.y);
      }
      *reinterpret_cast<float2 *>(red + ty * kDS + 2 * tx) = x;
    }
    // ---- dq, then X, and what follows from each -------------------------------
    float2 bq[TM], cq[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int t = R::row(ty, i);
      bq[i] = cq[i] = make_float2(0.f, 0.f);
      if (t < valid && on) {
        bq[i] = load_pair<T>(a.B + (tok0 + t) * d.D + dd);
        cq[i] = load_pair<T>(a.C + (tok0 + t) * d.D + dd);
      }
    }
    float acc[TM][2];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i][0] = acc[i][1] = 0.f;
    mm_kn<TM, 2>(acc, 0, p4, [&](int i) { return dYs + R::row(ty, i) * LP; },
                 [&](int k, int e) { return Zs + prow4<TP>(k, e) * kLdD + 2 * tx; });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      acc[i][0] *= el[i];
      acc[i][1] *= el[i];
    }
    mm_kn<TM, 2>(acc, 0, (R::warp_max() + 4) & ~3, [&](int i) { return dSs + R::row(ty, i) * LL; },
                 [&](int k, int e) { return Ks + (k + e) * kLdD + 2 * tx; });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int t = R::row(ty, i);
      const float2 dq = make_float2(fmaf(wv[t], km.x, acc[i][0]), fmaf(wv[t], km.y, acc[i][1]));
      const float2 dc = cmadd(ph[t], dq, cmul(cscale(kc[t], gd[t]), bq[i]));
      pgA[i] = cmadd(cq[i], cconj(dc), pgA[i]);
      if (t < valid && on) store_pair<T>(a.dC + (tok0 + t) * d.D + dd, dc);
      acc[i][0] = acc[i][1] = 0.f;
    }
    mm_kn<TM, 2>(acc, 0, p4, [&](int i) { return Us + R::row(ty, i) * LP; },
                 [&](int k, int e) { return Ls + prow4<TP>(k, e) * kLdD + 2 * tx; });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      acc[i][0] *= es[i];
      acc[i][1] *= es[i];
    }
    mm_mn<L, 2>(acc, R::warp_min(), L, [&](int k) { return dSs + k * LL + R::row(ty, 0); },
                [&](int k) { return Qs + k * kLdD + 2 * tx; });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int t = R::row(ty, i);
      const float2 X = make_float2(acc[i][0], acc[i][1]);
      const float2 db = cmadd(cconj(gk[t]), X, cmul(cscale(cconj(kc[t]), gd[t]), cq[i]));
      pP[i] = cmadd(cconj(bq[i]), X, pP[i]);
      if (t < valid && on) store_pair<T>(a.dB + (tok0 + t) * d.D + dd, db);
    }
    __syncthreads();
    if (tid < 16 && on) {  // dB_{-1} = conj(k^p_0) xi,  dk^p_0 += conj(b_{-1}) xi
      float2 x = make_float2(0.f, 0.f);
#pragma unroll
      for (int g = 0; g < 16; ++g) x = cadd(x, *reinterpret_cast<const float2 *>(red + g * kDS + 2 * tid));
      const float2 xi = cmul(ph[0], x);
      *reinterpret_cast<float2 *>(cB + dd) = cmul(cconj(kp[0]), xi);
      dkp0 = cmadd(cconj(bm), xi, dkp0);
    }
  }

  // ---- per-token sums -------------------------------------------------------
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = ty + 16 * i, t = R::row(ty, i);
    const float2 s0 = group_sum<16>(acc_bc[i]), s1 = group_sum<16>(make_float2(acc_s[i], 0.f));
    const float2 s2 = group_sum<16>(pgA[i]), s3 = group_sum<16>(pP[i]);
    if (tx == 0) {
      bc[r] = s0;
      sg[r] = expf(lp[r] - lp[0]) * s1.x;
      gA[t] = s2;
      bX[t] = cmul(ph[min(t + 1, L - 1)], s3);  // conj(b_s) xi_s
    }
  }
  acc_du += __shfl_xor_sync(0xffffffffu, acc_du, 1);
  acc_du += __shfl_xor_sync(0xffffffffu, acc_du, 2);
  if (tid < 64 * TP && (tid & 3) == 0) duc[tid >> 2] = es0 * acc_du;
  if (tid < 32) {
    const float2 s = group_sum<16>(dkp0);
    if (tid == 0) misc[0] = s;
  }
  __syncthreads();
  // ---- S' (forward scores) into shared memory; dU -----------------------------
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int t = R::row(ty, i);
#pragma unroll
    for (int j = 0; j < TM; ++j) {
      const int s = tx + 16 * j;
      float v = 0.f;
      if (s < t) v = S[i][j] * expf(lp[t] - lp[s + 1]);
      else if (s == t) v = kc[t].x * bc[t].x + kc[t].y * bc[t].y;  // Re(k^c_t conj(bc_t))
      dSs[t * LL + s] = v;
    }
#pragma unroll
    for (int j = 0; j < TP; ++j) dU[i][j] *= es[i];
  }
  // dU carried to the token before the chunk, by ty: sum_t sigma_t dY_t (the operand slabs are free)
  float *red2 = Qs;  // [16][16 TP]
#pragma unroll
  for (int e = 0; e < TP; ++e) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < TM; ++i) s = fmaf(sg[ty + 16 * i], dYs[(ty + 16 * i) * LP + TP * tx + e], s);
    red2[ty * 16 * TP + TP * tx + e] = s;
  }
  // ---- dK and the per-token terms of dM ------------------------------------------
  for (int t = tid; t < L; t += kThreads) {
    float2 dkc = cscale(bc[t], gd[t]);
    dkc = cadd(dkc, t + 1 < L ? cmul(cconj(mraw[t + 1]), bX[t]) : bX[t]);
    const float2 dkp = (t == 0) ? misc[0] : bX[t - 1];
    if (t < valid) *reinterpret_cast<float4 *>(a.dK + (tok0 + t) * 4) = make_float4(dkp.x, dkp.y, dkc.x, dkc.y);
    float2 g = csub(gA[t], cadd(cmul(cconj(kc[t]), dkc), cmul(cconj(kp[t]), dkp)));
    if (t == L - 1) {
      const float *zd = a.zdot + ((size_t)bh * d.NC + c) * 2;
      g = cadd(g, make_float2(zd[0], zd[1]));
    }
    gsum[t] = g;
  }
  __syncthreads();
  mm_mn<L, TP>(dU, R::warp_min(), L, [&](int k) { return dSs + k * LL + R::row(ty, 0); },
               [&](int k) { return dYs + k * LP + TP * tx; });
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int s = R::row(ty, i);
    if (s < valid) store_head<T, TP>(a.dU + (tok0 + s) * d.P, TP * tx, d.P, dU[i]);
  }
  if (tid >= kThreads - 16 * TP) {
    const int p = tid - (kThreads - 16 * TP);
    float s = duc[p];
#pragma unroll
    for (int g = 0; g < 16; ++g) s += red2[g * 16 * TP + p];
    if (p < d.P) a.carryU[((size_t)bh * d.NC + c) * d.P + p] = s;
  }
  // dM_t = (sum_{tau >= t} g_tau) m_t / |m_t|^2: suffix sum by one warp, adjacent tokens per lane
  if (tid < 32) {
    constexpr int PER = (L + 31) / 32;
    float2 loc[PER], run = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = PER - 1; i >= 0; --i) {
      const int t = tid * PER + i;
      if (t < L) run = cadd(run, gsum[t]);
      loc[i] = run;
    }
    float2 incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float ox = __shfl_down_sync(0xffffffffu, incl.x, off), oy = __shfl_down_sync(0xffffffffu, incl.y, off);
      if (tid + off < 32) incl = cadd(incl, make_float2(ox, oy));
    }
    float2 above = make_float2(__shfl_down_sync(0xffffffffu, incl.x, 1), __shfl_down_sync(0xffffffffu, incl.y, 1));
    if (tid == 31) above = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int t = tid * PER + i;
      if (t < valid && t < L) {
        const float2 m = mraw[t];
        const float inv = 1.f / (m.x * m.x + m.y * m.y);
        *reinterpret_cast<float2 *>(a.dM + (tok0 + t) * 2) = cscale(cmul(cadd(loc[i], above), m), inv);
      }
    }
  }
}

}  // namespace slx
