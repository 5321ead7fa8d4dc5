// One-token mixer decode step for sm_100a: scan prep of the token, one step of the
// recurrence on the carried state, skip and gate, in one kernel.
//
// Mirrors SLinOSSMixer._decode_step_reference (slinoss/layers/mixer.py:714-748) and the
// contract of mixer_decode_step_cute (slinoss/ops/v2x2ssd/cute/decode.py:117-149) without
// its shape restrictions (that kernel takes P = 64, N = 64, batch in {1,2,4,8,16} only):
//   (rho, k^p, k^c) = coefficient map(params + bias)              (prep_coef.cuh)
//   b, c            = interleave(rms_norm(bc) * scale), rounded to the activation dtype
//   z'[p][n]        = rho z[p][n] + k^p u_prev[p] b_prev[n] + k^c u[p] b[n]
//   y[p]            = sum_n Re(conj(c[n]) z'[p][n])
//   out[p]          = (y[p] + skip[p] u[p]) * silu(gate[p])
// The fp32 state (P x 2N) is the only large operand: a streaming warp owns four of every 32 rows, reads and
// writes them with 16-byte accesses (a row is contiguous) and reduces their y[p] by shuffles, so there is no
// cross-warp reduction and no atomics.
// The step is bound by HBM: 2 * P * 2N * 4 bytes per (batch, head).  The CTAs that fit the GPU
// walk over the heads: eight warps stream states, four others meanwhile prepare the operands of
// the next head (a serial chain of norms and the coefficient map, as long as the streaming
// itself) and finish the outputs of the last.  The state comes through shared memory by
// asynchronous copies, each thread reading back only what it copied itself, and the requests
// run ahead into the next head, so that the loads never stop.
// Batch 256, 32 heads, P 64, 2N 256: 238 us (4.5 TB/s) with a CTA per head that loaded four rows per
// warp at a time after its parameters -> 203 us (5.3 TB/s); 8 heads of 2N 128: 6.4 -> 6.5 us.
// A CTA per head with all of its state requested first took 311 us: the chain of the parameters
// was then exposed three CTAs deep.  Three CTAs per SM of three steps each are the optimum of
// {2, 3, 4} x {2, 3, 4}: fewer CTAs leave the writes uneven, four do not leave the registers.
#include "common.cuh"
#include "prep_coef.cuh"

namespace slx {

struct DecodeDims {
  int batch, H, P, N, normalize;
  long long vs, ps, bs, gs;  // elements between batches of value, params, bc, gate
  int skip_dtype;
};

constexpr int kDecodeWarps = 8;                           // warps that stream the state
constexpr int kDecodeStream = 32 * kDecodeWarps;
constexpr int kDecodePrep = 128;                          // threads that prepare the next and finish the last head
constexpr int kDecodeThreads = kDecodeStream + kDecodePrep;
constexpr int kDecodeRows = 4;                            // rows of a step, per warp
constexpr int kDecodeSteps = 3;                           // steps requested ahead
constexpr int kDecodeRing = 16 * kDecodeSteps * kDecodeRows * kDecodeStream;

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void decode_prep_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kDecodePrep) : "memory"); }

// One head's operands in shared memory, two of them in turn
struct DecodeBuf {
  float *c, *kb, *kbp;                // [D] c, k^c b, k^p b_prev
  float *u, *up, *y, *gate, *skip;    // [P]
  float2 *rho;                        // [1]
  float *rstd;                        // [4]
  __device__ DecodeBuf(float *base, int D, int P) {
    c = base; kb = c + D; kbp = kb + D;
    u = kbp + D; up = u + P; y = up + P; gate = y + P; skip = gate + P;
    rstd = skip + P + P % 2; rho = reinterpret_cast<float2 *>(rstd + 4);
  }
};
__host__ __device__ inline size_t decode_buf_floats(int D, int P) { return ((size_t)3 * D + 5 * P + 7 + 3) / 4 * 4; }

template <typename T>
__global__ void __launch_bounds__(kDecodeThreads, 3) decode_step_kernel(
    const T *__restrict__ value, const T *__restrict__ params, const T *__restrict__ bc, const T *__restrict__ gate,
    const void *__restrict__ skip, PrepParams pp, const float *state_in,
    const T *b_prev, const T *u_prev, T *__restrict__ out, float *state_out, T *b_last, T *u_last, DecodeDims d,
    PrepHyper hp) {
  extern __shared__ __align__(16) float sm[];
  const int D = 2 * d.N, n_items = D / 4, n_heads = d.batch * d.H;
  const int ring_floats = state_in ? kDecodeRing / 4 : 0;
  const DecodeBuf buf0(sm + ring_floats, D, d.P), buf1(sm + ring_floats + decode_buf_floats(D, d.P), D, d.P);
  __shared__ float2 coef[3 * 32];  // rho, k^p, k^c of up to 32 of the CTA's heads
  const int tid = threadIdx.x;
  const bool streams = tid < kDecodeStream;
  const int lane = tid & 31, warp = tid >> 5;

  // ---- state requests of a streaming thread.  Step = (head, rows ip + 8 r of this warp, item iq of every lane), the
  // item fastest; they run ahead of the steps that are worked on, into the next head
  float4 *ring = reinterpret_cast<float4 *>(sm) + tid;  // [steps][rows][threads]
  int ih = blockIdx.x, ip = kDecodeRows * warp, iq = lane, islot = 0;
  auto request = [&]() {
    if (state_in && ih < n_heads && iq < n_items) {
      const float *zin = state_in + (size_t)ih * d.P * D + 4 * iq;
#pragma unroll
      for (int r = 0; r < kDecodeRows; ++r) {
        const int p = ip + r;
        if (p < d.P) cp_async16(ring + (islot * kDecodeRows + r) * kDecodeStream, zin + (size_t)p * D);
      }
    }
    cp_async_commit();
    islot = islot + 1 == kDecodeSteps ? 0 : islot + 1;
    iq += 32;
    if (iq - lane >= n_items) {
      iq = lane;
      ip += kDecodeWarps * kDecodeRows;
      if (ip - kDecodeRows * warp >= d.P) {
        ip = kDecodeRows * warp;
        ih += gridDim.x;
      }
    }
  };

  // ---- operands of one head, by the preparing threads
  const int t = tid - kDecodeStream;
  auto prepare = [&](int bh, int k, const DecodeBuf &s) {  // the CTA's k-th
    // the coefficient map is a long serial chain: a lane per head, for this and the 31 after it (in the last warp, which
    // has the fewest other loads to wait for)
    const int ahead = bh + (int)gridDim.x * lane;
    if ((k & 31) == 0 && t >= kDecodePrep - 32 && ahead < n_heads) {
      const int h = ahead % d.H, b_ = ahead / d.H;
      float p[13];
#pragma unroll
      for (int i = 0; i < 13; ++i) p[i] = to_f(params[(size_t)b_ * d.ps + (size_t)h * 13 + i]);
      add_bias13(pp, h, p);
      const CoefOut o = coef_forward(p, hp, nullptr);
      coef[3 * lane] = o.rho;
      coef[3 * lane + 1] = o.kp;
      coef[3 * lane + 2] = o.kc;
    }
    const int h = bh % d.H, b_ = bh / d.H;
    const T *bcr = bc + (size_t)b_ * d.bs + (size_t)h * 4 * d.N;
    float raw[4], scl[4];
    float2 bp = make_float2(0.f, 0.f);
    auto load_n = [&](int n) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        raw[j] = to_f(bcr[j * d.N + n]);
        scl[j] = d.normalize ? load_as_f(scale_plane(pp, j), pp.dtype, scale_index(pp, h, j, d.N, n)) : 1.f;
      }
      if (b_prev) bp = make_float2(to_f(b_prev[(size_t)bh * D + 2 * n]), to_f(b_prev[(size_t)bh * D + 2 * n + 1]));
    };
    if (t < d.N) load_n(t);  // requested before anything is waited for
    for (int p = t; p < d.P; p += kDecodePrep) {
      const float u = to_f(value[(size_t)b_ * d.vs + (size_t)h * d.P + p]);
      s.u[p] = u;
      s.up[p] = u_prev ? to_f(u_prev[(size_t)bh * d.P + p]) : 0.f;
      s.gate[p] = to_f(gate[(size_t)b_ * d.gs + (size_t)h * d.P + p]);
      // skip takes part rounded to the activation dtype, whatever it is stored in
      s.skip[p] = to_f(from_f<T>(load_as_f(skip, d.skip_dtype, (size_t)h * d.P + p)));
      if (u_last) u_last[(size_t)bh * d.P + p] = from_f<T>(u);
    }
    // rms-norm statistics: warp j owns plane j of bc
    float ss = 0.f;
    for (int n = lane; n < d.N; n += 32) {
      const float v = to_f(bcr[(t >> 5) * d.N + n]);
      ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (lane == 0) s.rstd[t >> 5] = d.normalize ? rsqrtf(ss / (float)d.N + 1e-5f) : 1.f;
    decode_prep_sync();
    const float2 kp = coef[3 * (k & 31) + 1], kc = coef[3 * (k & 31) + 2];
    if (t == 0) s.rho[0] = coef[3 * (k & 31)];
    for (int n = t; n < d.N; n += kDecodePrep) {
      if (n != t) load_n(n);
      float y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v = raw[j];
        if (d.normalize) v = (v * s.rstd[j]) * scl[j];
        y[j] = to_f(from_f<T>(v));  // the reference casts the normalised rows back before the scan
      }
      const float2 b = make_float2(y[0], y[1]);
      *reinterpret_cast<float2 *>(s.c + 2 * n) = make_float2(y[2], y[3]);
      *reinterpret_cast<float2 *>(s.kb + 2 * n) = cmul(kc, b);
      *reinterpret_cast<float2 *>(s.kbp + 2 * n) = cmul(kp, bp);
      if (b_last) {
        b_last[(size_t)bh * D + 2 * n] = from_f<T>(b.x);
        b_last[(size_t)bh * D + 2 * n + 1] = from_f<T>(b.y);
      }
    }
  };
  auto finish = [&](int bh, const DecodeBuf &s) {
    for (int p = t; p < d.P; p += kDecodePrep) {
      const float g = s.gate[p], y = s.y[p] + s.skip[p] * s.u[p];
      out[(size_t)bh * d.P + p] = from_f<T>(y * (g / (1.f + expf(-g))));
    }
  };

  if (streams) {
#pragma unroll
    for (int k = 0; k < kDecodeSteps; ++k) request();
  } else {
    prepare(blockIdx.x, 0, buf0);
  }
  __syncthreads();
  int slot = 0, it = 0, bh = blockIdx.x;
  for (; bh < n_heads; bh += gridDim.x, ++it) {
    const DecodeBuf &s = it & 1 ? buf1 : buf0;
    if (streams) {
      // warp w owns rows 4 w .. 4 w + 3 of every 32; a lane owns the float4 items q = lane + 32 i
      const float2 m = s.rho[0];
      float *zout = state_out + (size_t)bh * d.P * D;
      for (int p0 = kDecodeRows * warp; p0 - kDecodeRows * warp < d.P; p0 += kDecodeWarps * kDecodeRows) {
        float acc[kDecodeRows];
#pragma unroll
        for (int r = 0; r < kDecodeRows; ++r) acc[r] = 0.f;
        for (int q0 = lane; q0 - lane < n_items; q0 += 32) {
          cp_async_wait<kDecodeSteps - 1>();  // this thread's own copies of the step
          float4 z[kDecodeRows];
#pragma unroll
          for (int r = 0; r < kDecodeRows; ++r)
            z[r] = state_in ? ring[(slot * kDecodeRows + r) * kDecodeStream] : make_float4(0.f, 0.f, 0.f, 0.f);
          slot = slot + 1 == kDecodeSteps ? 0 : slot + 1;
          request();
          if (q0 >= n_items) continue;
          const float4 vkb = *reinterpret_cast<const float4 *>(s.kb + 4 * q0);
          const float4 vkbp = *reinterpret_cast<const float4 *>(s.kbp + 4 * q0);
          const float4 vc = *reinterpret_cast<const float4 *>(s.c + 4 * q0);
#pragma unroll
          for (int r = 0; r < kDecodeRows; ++r) {
            const int p = p0 + r;
            if (p < d.P) {
              const float u = s.u[p], up = s.up[p];
              float4 o;
              o.x = fmaf(m.x, z[r].x, fmaf(-m.y, z[r].y, fmaf(up, vkbp.x, u * vkb.x)));
              o.y = fmaf(m.x, z[r].y, fmaf(m.y, z[r].x, fmaf(up, vkbp.y, u * vkb.y)));
              o.z = fmaf(m.x, z[r].z, fmaf(-m.y, z[r].w, fmaf(up, vkbp.z, u * vkb.z)));
              o.w = fmaf(m.x, z[r].w, fmaf(m.y, z[r].z, fmaf(up, vkbp.w, u * vkb.w)));
              *reinterpret_cast<float4 *>(zout + (size_t)p * D + 4 * q0) = o;
              acc[r] += fmaf(vc.x, o.x, fmaf(vc.y, o.y, fmaf(vc.z, o.z, vc.w * o.w)));
            }
          }
        }
#pragma unroll
        for (int r = 0; r < kDecodeRows; ++r) {
          float a = acc[r];
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
          const int p = p0 + r;
          if (lane == 0 && p < d.P) s.y[p] = a;
        }
      }
    } else {
      const DecodeBuf &o = it & 1 ? buf0 : buf1;
      if (it > 0) {
        finish(bh - gridDim.x, o);
        decode_prep_sync();  // the buffer is free
      }
      if (bh + (int)gridDim.x < n_heads) prepare(bh + gridDim.x, it + 1, o);
    }
    __syncthreads();
  }
  if (!streams && it > 0) finish(bh - gridDim.x, (it - 1) & 1 ? buf1 : buf0);
  cp_async_wait<0>();
}

}  // namespace slx

using namespace slx;

static int decode_impl(const slx_decode_shape *s, const void *value, const void *params, const void *bc,
                       const void *gate, const int64_t *strides, const void *skip, int skip_dtype, const PrepParams &pp,
                       const float *state_in, const void *b_prev, const void *u_prev, void *out, float *state_out,
                       void *b_last, void *u_last, void *stream) {
  SLX_REQUIRE(s->batch > 0 && s->heads > 0 && s->P > 0 && s->N > 0, SLX_E_SHAPE, "decode_step: sizes must be positive");
  SLX_REQUIRE(s->N % 2 == 0, SLX_E_UNSUPPORTED, "decode_step: N=%d must be even (16-byte state accesses)", s->N);
  SLX_REQUIRE(s->dtype == SLX_F32 || s->dtype == SLX_BF16 || s->dtype == SLX_F16, SLX_E_DTYPE,
              "decode_step: unknown dtype code %d", s->dtype);
  SLX_REQUIRE(value && params && bc && gate && skip && out && state_out, SLX_E_NULL, "decode_step: NULL tensor");
  SLX_REQUIRE(!s->normalize_bc || (pp.b_scale && pp.c_scale), SLX_E_NULL,
              "decode_step: scale is NULL with normalize_bc set");
  SLX_REQUIRE((b_prev == nullptr) == (u_prev == nullptr), SLX_E_NULL,
              "decode_step: b_prev and u_prev go together");
  SLX_REQUIRE((reinterpret_cast<uintptr_t>(state_out) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(state_in) & 15) == 0,
              SLX_E_UNSUPPORTED, "decode_step: state pointers must be 16-byte aligned");
  DecodeDims d{s->batch, s->heads, s->P, s->N, s->normalize_bc,
               strides ? strides[0] : (long long)s->heads * s->P, strides ? strides[1] : (long long)s->heads * 13,
               strides ? strides[2] : (long long)s->heads * 4 * s->N, strides ? strides[3] : (long long)s->heads * s->P,
               skip_dtype};
  PrepHyper hp;
  hp.dt_min = s->dt_min; hp.dt_max = s->dt_max; hp.r_min = s->r_min; hp.r_max = s->r_max;
  hp.theta_bound = s->theta_bound; hp.k_max = s->k_max;
  {
    float e = s->eps > 1e-12f ? s->eps : 1e-12f;
    float thr = sqrtf(e);
    if (thr < 1e-4f) thr = 1e-4f;
    hp.z_thr2 = thr * thr;
  }
  const size_t vecs = sizeof(float) * ((size_t)8 * s->N + 3 * (size_t)s->P + 16);
  SLX_REQUIRE(vecs <= 48 * 1024, SLX_E_UNSUPPORTED, "decode_step: N=%d, P=%d need %zu bytes of shared memory",
              s->N, s->P, vecs);
  const size_t smem = (state_in ? kDecodeRing : 0) + 2 * sizeof(float) * decode_buf_floats(2 * s->N, s->P);
  const long long heads = (long long)s->batch * s->heads;
  SLX_REQUIRE(heads <= 2147483647LL, SLX_E_UNSUPPORTED, "decode_step: batch*heads too large");
  cudaStream_t st = as_stream(stream);
  auto launch = [&](auto t) {
    using TT = decltype(t);
    auto kern = decode_step_kernel<TT>;
    if (int rc = ensure_dyn_smem(kern, smem)) return rc;
    const long resident = resident_ctas(kern, kDecodeThreads, smem);
    const unsigned grid = (unsigned)(resident > 0 && resident < heads ? resident : heads);
    kern<<<grid, kDecodeThreads, smem, st>>>(
        (const TT *)value, (const TT *)params, (const TT *)bc, (const TT *)gate, skip, pp, state_in,
        (const TT *)b_prev, (const TT *)u_prev, (TT *)out, state_out, (TT *)b_last, (TT *)u_last, d, hp);
    return check_launch("decode_step");
  };
  if (s->dtype == SLX_F32) return launch(float());
  return s->dtype == SLX_BF16 ? launch(__nv_bfloat16()) : launch(__half());
}

extern "C" int slx_decode_step(const slx_decode_shape *s, const void *value, const void *params, const void *bc,
                               const void *gate, const void *skip, const float *bias, const float *scale,
                               const float *state_in, const void *b_prev, const void *u_prev, void *out,
                               float *state_out, void *b_last, void *u_last, void *stream) {
  SLX_REQUIRE(s != nullptr, SLX_E_NULL, "decode_step: shape is NULL");
  SLX_REQUIRE(bias != nullptr, SLX_E_NULL, "decode_step: NULL tensor");
  constexpr int kSlot[7] = {0, 1, 2, 5, 6, 7, 8};
  PrepParams pp{};
  for (int k = 0; k < 7; ++k) pp.bias[k] = bias + kSlot[k];
  pp.b_scale = scale;
  pp.c_scale = scale ? scale + 2 * s->N : nullptr;
  pp.dtype = SLX_F32;
  pp.bias_stride = 13;
  pp.scale_stride = 4LL * s->N;
  return decode_impl(s, value, params, bc, gate, nullptr, skip, s->dtype, pp, state_in, b_prev, u_prev, out, state_out,
                     b_last, u_last, stream);
}

extern "C" int slx_decode_step_params(const slx_decode_shape *s, const void *value, const void *params, const void *bc,
                                      const void *gate, const int64_t *batch_strides, const void *skip,
                                      int32_t skip_dtype, const slx_prep_params *p, const float *state_in,
                                      const void *b_prev, const void *u_prev, void *out, float *state_out, void *b_last,
                                      void *u_last, void *stream) {
  SLX_REQUIRE(s != nullptr && p != nullptr, SLX_E_NULL, "decode_step: shape or params is NULL");
  SLX_REQUIRE(p->dtype >= SLX_F32 && p->dtype <= SLX_F16 && skip_dtype >= SLX_F32 && skip_dtype <= SLX_F16, SLX_E_DTYPE,
              "decode_step: bad parameter dtype %d or %d", p->dtype, skip_dtype);
  PrepParams pp{};
  for (int k = 0; k < 7; ++k) {
    SLX_REQUIRE(p->bias[k] != nullptr, SLX_E_NULL, "decode_step: bias %d is NULL", k);
    pp.bias[k] = p->bias[k];
  }
  pp.b_scale = p->b_scale;
  pp.c_scale = p->c_scale;
  pp.dtype = p->dtype;
  pp.bias_stride = 1;
  pp.scale_stride = 2LL * s->N;
  return decode_impl(s, value, params, bc, gate, batch_strides, skip, skip_dtype, pp, state_in, b_prev, u_prev, out,
                     state_out, b_last, u_last, stream);
}
