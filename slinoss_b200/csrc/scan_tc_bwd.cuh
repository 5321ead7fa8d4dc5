// Tensor-core per-chunk backward of the v2x2ssd scan (chunk 128, P 64, half
// inputs, fp32 state).  Same mathematics as chunk_scan_bwd_kernel in
// scan_simt.cuh; every contraction runs on tcgen05 with fp32 accumulators in
// tensor memory.  One CTA per (chunk, batch*head): 8 warps, two CTAs per SM, or, in launches of at most one CTA per SM
// (LONE), 16 warps.
//
// Phases are taken relative to the end of the chunk, f_t = phi_t conj(phi_{L-1}), so that Lambda, Z0, U and dY enter
// their products as they are stored.  Operands per slab of the state, 32 columns or LONE 64 (half precision, every one
// rounded once from fp32 or as it is stored):
//   Q_t = c_t conj(f_t),  kappa_s = gamma_s b_s conj(f_{s+1}),  Z0,  Lambda
// and per chunk  dS' = decay * (dY U^T),  dY,  U.  With es_s = p_{L-1}/p_{s+1} in magnitude, p_t = exp(lp_t) phi_t:
//   dC_t = f_t (dS' kappa)_t + p_t (dY Z0)_t + (k^c_t G_tt) b_t
//   xi_s = (dS'^T Q)_s + es_s (U Lambda)_s,   dB_s = conj(gamma_s) f_{s+1} xi_s + conj(k^c_s G_ss) c_s
//   dU   = S'^T dY + es (kappa Lambda^T)
// Scales and rotations of a row are applied to the fp32 accumulators, never to an operand that is rounded already.
//
// Slot 127 of the source axis (U, kappa) holds the token in front of the chunk: the merged-tap column of token 127 is
// empty (no query follows it), and that row of dS', dS'^T Q, U Lambda, kappa Lambda^T and S'^T dY is then what the carry
// gradients need.  Token 127's own increment path, u_127 . Lambda and (k^c b_127) . Lambda, and its diagonal terms are
// summed on the CUDA cores.
//
// Tensor-memory map (256 fp32 columns):
//   [  0,128)  G = dY U^T, then S^T = kappa Q^T       (accumulated over the slabs)
//   [128,192)  kappa Lambda^T                         (accumulated over the slabs)
//   [192,224)  dS'^T Q of a slab, then dS' kappa      [224,256)  U Lambda, then dY Z0;  [192,256) at the end S'^T dY
// LONE: 512 columns, [192,256) dS'^T Q, [256,320) U Lambda, [320,384) dS' kappa, [384,448) dY Z0.
//
// Columns of kappa, Q, Lambda and Z0 are stored (re, re, re, re, im, im, im, im) inside each group of four complex
// values: sums over the state do not see the order, and the accumulators then hold real and imaginary parts of two
// values side by side, which is what the packed fp32 arithmetic (two fmas per instruction) takes.
//
// What bounds it: neither HBM (46 %) nor the tensor pipe (12 %) but instruction issue and the latencies between a
// chunk's phases (loads and prefix, slabs, tail).  8192 chunks of D 256: 1.052 ms.  One CTA of 16 worker warps per SM
// with 64-column slabs and two buffers for every operand took 1.205 ms: its phases followed one another and nothing
// filled their latencies.  Two CTAs of 8 warps run different phases at the same time.  They fit because the slabs are 32
// columns wide with one buffer, dS'^T Q / U Lambda and dS' kappa / dY Z0 take turns in the same 64 accumulator columns,
// and dC / dB leave from registers (whole 32-byte sectors).  Measured on the way: a ninth warp that issues the products
// leaves 96 registers to a thread, and the spills cost more than the issuing (1.097 against 0.997 ms); one thread that
// waits for the products and a CTA barrier behind it 1.198 against 1.070 ms.
//
// LONE: where a launch has no more chunks than SMs the second CTA is missing, and the latencies of one chain show.  Twice
// the threads and slabs of 64 columns halve the steps of that chain, and accumulators of their own for all four products of
// a slab let them be issued together, with one CTA barrier per slab.  us, 8 warps and 32 columns / LONE: 148 chunks of D 256
// 33.4 / 26.2, of D 128 23.3 / 18.7, 64 of D 64 17.6 / 14.3, 16 of D 256 27.3 / 22.5 (one CTA of 16 warps per SM with double
// buffers: 23.6, 16.8, 13.6, 21.1).  16 warps with 32 columns 29.9, the same with accumulators of their own 29.7 (148 of D 256).
//
// PREV32: the streaming rows are fp32.  The tile then holds u_{-1} rounded, and its products with dY and Lambda get what
// that lost from the CUDA cores, as u_{-1} enters dB_prev, dK and dM in fp32.  An instantiation of its own: as a branch it
// costs every launch (8192 chunks of D 256: 1.064 against 1.050 ms).
//
// Thread mapping: thread = (row 32*(warp%4)+lane, 16-byte cells 2*(warp/4) and +1 of the slab), the tensor-memory
// lane mapping, for staging and epilogue alike, so that the raw b, c of a cell stay in registers from one to the other.
#pragma once

#include "scan_tc.cuh"

namespace slx {

// tensor maps of the raw C and B operands: (D, T, BH), boxes of a slab x 128 tokens, 64-byte swizzle (LONE: 128-byte)
struct alignas(64) ScanBwdMaps {
  CUtensorMap C, B;
};

constexpr uint32_t bwd_scalars(bool lone) { return lone ? 147456 : 106496; }
constexpr size_t scan_bwd_tc_smem_bytes(bool lone, bool prev32) {
  return bwd_scalars(lone) + 8320 + (lone ? 9216 : 0) + (prev32 ? 256 : 0);
}
constexpr int kTmR = 128, kTmX = 192, kTmU = kTmX;  // accumulator columns (G / S^T at 0)

// (a + i b) * cell, packed as four real parts and four imaginary parts
template <typename T>
__device__ __forceinline__ uint4 rotate_cell_split(const CellF &c, float a, float b) {
  uint4 out;
  uint32_t *o = reinterpret_cast<uint32_t *>(&out);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float2 re = __ffma2_rn(both(a), c.re[q], __fmul2_rn(both(-b), c.im[q]));
    const float2 im = __ffma2_rn(both(a), c.im[q], __fmul2_rn(both(b), c.re[q]));
    o[q] = umma::pack2(re.x, re.y, T());
    o[2 + q] = umma::pack2(im.x, im.y, T());
  }
  return out;
}
__device__ __forceinline__ uint4 split_cell(uint4 v) {  // (re, im) pairs -> four real parts, four imaginary parts
  return make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.x, v.y, 0x7632),
                    __byte_perm(v.z, v.w, 0x7632));
}
template <typename T>
__device__ __forceinline__ CellF unpack_cell_split(uint4 v) {  // of a cell packed by rotate_cell_split
  return CellF{{umma::unpack2(v.x, T()), umma::unpack2(v.y, T())}, {umma::unpack2(v.z, T()), umma::unpack2(v.w, T())}};
}
__device__ __forceinline__ float2 tm_pair(const uint32_t *r) {
  return make_float2(__uint_as_float(r[0]), __uint_as_float(r[1]));
}

template <typename T, bool PREV32, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) chunk_scan_bwd_tc_kernel(ScanBwdArgs<T> a,
                                                                              const __grid_constant__ ScanBwdMaps maps) {
  constexpr int L = kTcL, P = kTcP;
  constexpr bool LONE = THREADS == 512;
  constexpr int COLS = THREADS / 128, PARTS = 4 / COLS;  // threads per row; passes over the 128 columns of a score tile
  constexpr int SW = 16 * COLS;                          // columns of a slab: two 16-byte cells per thread and row
  constexpr uint32_t kTmUL = kTmX + SW, kTmX2 = LONE ? kTmX + 2 * SW : kTmX, kTmUL2 = LONE ? kTmX + 3 * SW : kTmUL;
  // shared memory from 65536 on: kappa, Q, Lambda, Z0, raw C, raw B, scalars
  constexpr uint32_t oK = 65536, oQ = oK + 256 * SW, oLm = oQ + 256 * SW, oZ = oLm + 128 * SW, oC = oZ + 128 * SW,
                     oB = oC + 256 * SW, oS = oB + 256 * SW;
  static_assert(oS == bwd_scalars(LONE), "shared-memory layout");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *base = smem_raw;
  unsigned char *tdY = base;                   // [t][p]
  unsigned char *tU = base + 16384;            // [s][p]
  unsigned char *tdS = base + 32768;           // 2 x [t][64 s]  dS', at the end 2 x [s][64 t]  S'^T
  unsigned char *tK = base + oK;               // [s][SW d]  kappa
  unsigned char *tQ = base + oQ;               // [t][SW d]  Q
  unsigned char *tLm = base + oLm;             // [p][SW d]  Lambda
  unsigned char *tZ = base + oZ;               // [p][SW d]  Z0
  unsigned char *sC = base + oC;               // raw C slab, by TMA; scratch of the tail
  unsigned char *sB = base + oB;               // raw B slab
  float *lp = reinterpret_cast<float *>(base + oS);
  float *tab = lp + L;                         // decay table of dS' (decay_table_entry), then of S'^T
  float *gd = tab + L;                         // G[t][t]
  float *um = gd + L;                          // 64   u_127
  float *duc = um + 64;                        // 64   (k^c b_127) . Lambda[p]
  float *xb = duc + 64;                        // 256  dS'^T Q of the token in front of the chunk
  float *ulf = xb + 256;                       // 256  u_127 . Lambda
  float *ulw = ulf + 256;                      // [8][32] per-warp partials of u_127 . Lambda
  float2 *mraw = reinterpret_cast<float2 *>(xb), *kc = reinterpret_cast<float2 *>(ulf),
         *kp = reinterpret_cast<float2 *>(ulw);  // until the rows' coefficients are formed
  float2 *ph = reinterpret_cast<float2 *>(ulw + 256);
  float2 *bm1 = ph + L;                        // 128  b_{-1}
  float2 *bh1 = bm1 + 128;                     // 128  k^c b_127
  float *more = reinterpret_cast<float *>(base + oS + 8320);  // LONE: 256, 2 x [16][64] partials of u_127 . Lambda
  // 256  U Lambda of the token in front of the chunk; without LONE over bh1, behind helper()'s reads
  float *ub = LONE ? more : reinterpret_cast<float *>(bh1);
  float2 *misc = bh1 + 128;                    // [0..3] dk^p_0, [4..7] sum conj(b_127) (u_127 . Lambda), by warp
  uint64_t *bars = reinterpret_cast<uint64_t *>(misc + 8);  // [0] first, [1] second products of a slab; [2] G, then
                                                            // S'^T dY; [3] raw slab by TMA
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 4);
  float *ulo = more + (LONE ? 2304 : 0);       // PREV32: 64  what u_{-1} loses in its tile
  static_assert(4 * (3 * 128 + 2 * 64 + 3 * 256) + 8 * 3 * 128 + 64 + 4 * 8 + 8 <= 8320, "shared-memory layout");
  // scratch of the tail, over the raw slabs
  float2 *pgs = reinterpret_cast<float2 *>(sC), *pbs = pgs + (COLS - 1) * L;  // gA, bX of the column parts behind the first
  float2 *pcs = pbs + (COLS - 1) * L, *bXs = pcs + COLS * L;                   // bc by column part; bX
  float2 *sums = bXs + L;  // [0..3] g by warp, [4..7] correction of slot 127 by warp

  const ScanDims d = a.d;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int t0 = c * L;
  const int valid = min(L, d.T - t0);
  const size_t tok0 = (size_t)bh * d.T + t0;
  const int NB = d.D / SW;
  const uint32_t bar0 = umma::smem_u32(bars), gbar = bar0 + 16, tbar = bar0 + 24;
  constexpr int fmt = umma::HalfFmt<T>::value;

#define SLX_STAMP(i) SLX_DIAG_STAMP(i)
  SLX_STAMP(0);
  // on this path the chunk-start states are stored in the activation dtype (api: slx_scan_starts_dtype)
  const T *z0 = reinterpret_cast<const T *>(a.starts) + ((size_t)bh * d.NC + c) * P * d.D;
  const T *lam = reinterpret_cast<const T *>(a.d_inc) + ((size_t)bh * d.NC + c) * P * d.D;  // same dtype as z0
  float2 mreg[4];  // the prefix warp's multipliers, requested ahead of the bulk copies
  if (warp == 2) chunk_prefix_load4(a.M + tok0 * 2, valid, mreg);
  // U and dY land in their tiles by asynchronous copy (rows past the chunk end are zero-filled)
  constexpr int ROWS = THREADS / 8;
  const int j8 = tid & 7, r8 = tid >> 3;
  uint4 ucell = make_uint4(0, 0, 0, 0);  // the thread that copies a cell of row 127: that cell of u_{-1}
#pragma unroll
  for (int i = 0; i < L / ROWS; ++i) {
    const int r = r8 + ROWS * i;
    const int rr = r < valid ? r : 0;
    const uint32_t nbytes = r < valid ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(tU + umma::swz_off(r, j8))),
                 "l"(a.U + (tok0 + rr) * P + 8 * j8), "r"(nbytes)
                 : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(tdY + umma::swz_off(r, j8))),
                 "l"(a.dY + (tok0 + rr) * P + 8 * j8), "r"(nbytes)
                 : "memory");
  }
  if (r8 == ROWS - 1) {
    if (t0 > 0) {
      ucell = *reinterpret_cast<const uint4 *>(a.U + (tok0 - 1) * P + 8 * j8);
    } else if (a.Uprev) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = load_as_f(a.Uprev, a.prev_dtype, (size_t)bh * P + 8 * j8 + e);
      ucell = pack8<T>(v);
      if constexpr (PREV32) {
#pragma unroll
        for (int e = 0; e < 8; ++e) ulo[8 * j8 + e] = v[e] - to_f(from_f<T>(v[e]));
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // One raw (C, B) slab = two TMA boxes of [128 tokens][SW columns] into the swizzled staging tiles,
  // issued by one thread; tokens past the end of the sequence arrive as zeros.
  auto prefetch_cb = [&](int sl) {
    umma::fence_smem_to_async();  // the tiles' earlier (generic) readers are behind a barrier
    umma::mbar_expect_tx(tbar, 2u * 256u * SW);
    umma::tma_load_3d(umma::smem_u32(sC), &maps.C, sl * SW, t0, bh, tbar);
    umma::tma_load_3d(umma::smem_u32(sB), &maps.B, sl * SW, t0, bh, tbar);
  };
  if (tid == 0) {
    umma::mbar_init(bar0, 2);      // commits of issue_first
    umma::mbar_init(bar0 + 8, 3);  // and of issue_second
    umma::mbar_init(gbar, 1);
    umma::mbar_init(tbar, 1);
    umma::fence_mbar_init();
    umma::tma_prefetch_map(&maps.C);
    umma::tma_prefetch_map(&maps.B);
    prefetch_cb(0);
  }
  // Z0 / Lambda slab: one 8-value (16-byte) item per thread, prefetched into registers
  const int zp = tid / (SW / 8), zj = tid % (SW / 8);
  uint4 zr, lr;
  auto prefetch_zl = [&](int sl) {
    zr = *reinterpret_cast<const uint4 *>(z0 + (size_t)zp * d.D + sl * SW + 8 * zj);
    lr = *reinterpret_cast<const uint4 *>(lam + (size_t)zp * d.D + sl * SW + 8 * zj);
  };
  prefetch_zl(0);

  if (warp == 1) umma::tmem_alloc(tmem_slot, LONE ? 512 : 256);
  if (warp == 2) chunk_prefix_fast128(mreg, lp, ph, mraw, &g_scan_bad);
  if ((tid >> 7) == 1) {
    const int t = tid - 128;
    float2 vp = make_float2(0.f, 0.f), vc = vp;
    if (t < valid) {
      float4 k4 = *reinterpret_cast<const float4 *>(a.K + (tok0 + t) * 4);
      vp = make_float2(k4.x, k4.y);
      vc = make_float2(k4.z, k4.w);
    }
    kp[t] = vp;
    kc[t] = vc;
    if (t < d.N) {
      float2 bv = make_float2(0.f, 0.f), bl = bv;
      if (t0 > 0) bv = load_pair<T>(a.B + (tok0 - 1) * d.D + 2 * t);
      else if (a.Bprev) bv = load_as_f2(a.Bprev, a.prev_dtype, (size_t)bh * d.D + 2 * t);
      if (valid == L)
        bl = cmul(*reinterpret_cast<const float2 *>(a.K + (tok0 + L - 1) * 4 + 2),
                  load_pair<T>(a.B + (tok0 + L - 1) * d.D + 2 * t));
      bm1[t] = bv;
      bh1[t] = bl;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");  // U, dY tiles
  if (r8 == ROWS - 1) {  // source slot 127 is the token in front of the chunk; u_127 is kept aside
    uint4 *cell = reinterpret_cast<uint4 *>(tU + umma::swz_off(L - 1, j8));
    const uint4 own = *cell;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(&own);
#pragma unroll
    for (int e = 0; e < 4; ++e) *reinterpret_cast<float2 *>(um + 8 * j8 + 2 * e) = umma::unpack2(w[e], T());
    *cell = ucell;
  }
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  SLX_STAMP(1);
  // ---- the products --------------------------------------------------------------------------
  // Issuing a product takes about as long as the product (90 cycles), so several warps share it: nobody is held longer
  // than the products that every warp waits for take (8192 chunks: 1.059 ms, all by one thread 1.141).
  constexpr uint32_t id_km = umma::make_idesc(128, SW, false, true, fmt);
  constexpr uint32_t id_sq = umma::make_idesc(128, 128, false, false, fmt);
  const uint32_t sb = umma::smem_u32(base);
  // a slab tile as an operand: 64-byte rows (SW 32, one descriptor for both views) or 128-byte rows
  constexpr uint32_t kMN = LONE ? umma::kStepMN : umma::kStepMN64;
  auto mn_view = [&](uint32_t off) { return LONE ? umma::desc_mnmajor(sb + off, 0, 0) : umma::make_desc64(sb + off); };
  auto k_view = [&](uint32_t off) { return LONE ? umma::desc_kmajor(sb + off, 0) : umma::make_desc64(sb + off); };
  // (LONE: all five of a slab at its start, by warps that have no helper())
  auto issue_first = [&](int sl) {  // dS'^T Q (warp 0), U Lambda (warp 1)
    if (warp == (LONE ? 8 : 0)) {
      if (lane == 0) {
        umma::fence_after_sync();
        constexpr uint32_t id_mm = umma::make_idesc(128, SW, true, true, fmt);
        const uint64_t dSm = umma::desc_mnmajor(sb + 32768, 0, 16384u), dQ = mn_view(oQ);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma::mma_ss(tmem + kTmX, umma::desc_advance(dSm, umma::kStepMN * kk),
                       umma::desc_advance(dQ, kMN * kk), id_mm, kk != 0);
        umma::commit(bar0);
      }
      __syncwarp();
    } else if (warp == (LONE ? 9 : 1)) {
      if (lane == 0) {
        umma::fence_after_sync();
        const uint64_t dUk = umma::desc_kmajor(sb + 16384, 0), dLm = mn_view(oLm);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma::mma_ss(tmem + kTmUL, umma::desc_advance(dUk, umma::kStepK * kk),
                       umma::desc_advance(dLm, kMN * kk), id_km, kk != 0);
        umma::commit(bar0);
        if (sl > 0 && sl + 1 < NB) prefetch_cb(sl + 1);
      }
      __syncwarp();
    }
  };
  auto issue_second = [&](int sl) {  // dS' kappa (warp 5), dY Z0 (warp 6), S^T and kappa Lambda^T (warp 7)
    if (warp == (LONE ? 10 : 5)) {
      if (lane == 0) {
        umma::fence_after_sync();
        const uint64_t dSk = umma::desc_kmajor(sb + 32768, 0), dK = mn_view(oK);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma::mma_ss(tmem + kTmX2, umma::desc_advance(dSk, 16384u * (kk >> 2) + umma::kStepK * (kk & 3)),
                       umma::desc_advance(dK, kMN * kk), id_km, kk != 0);
        umma::commit(bar0 + 8);
      }
      __syncwarp();
    } else if (warp == (LONE ? 11 : 6)) {
      if (lane == 0) {
        umma::fence_after_sync();
        const uint64_t dYk = umma::desc_kmajor(sb, 0), dZ = mn_view(oZ);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma::mma_ss(tmem + kTmUL2, umma::desc_advance(dYk, umma::kStepK * kk),
                       umma::desc_advance(dZ, kMN * kk), id_km, kk != 0);
        umma::commit(bar0 + 8);
      }
      __syncwarp();
    } else if (warp == (LONE ? 12 : 7)) {
      if (lane == 0) {
        umma::fence_after_sync();
        constexpr uint32_t id_kk = umma::make_idesc(128, 64, false, false, fmt);
        const uint64_t dK = k_view(oK), dQ = k_view(oQ), dLm = k_view(oLm);
#pragma unroll
        for (int kk = 0; kk < SW / 16; ++kk) {
          umma::mma_ss(tmem, umma::desc_advance(dK, umma::kStepK * kk), umma::desc_advance(dQ, umma::kStepK * kk), id_sq,
                       (sl | kk) != 0);
          umma::mma_ss(tmem + kTmR, umma::desc_advance(dK, umma::kStepK * kk),
                       umma::desc_advance(dLm, umma::kStepK * kk), id_kk, (sl | kk) != 0);
        }
        umma::commit(bar0 + 8);
      }
      __syncwarp();
    }
  };
  if (warp == 0) {
    if (lane == 0) {
      const uint64_t dYk = umma::desc_kmajor(sb, 0), dUk = umma::desc_kmajor(sb + 16384, 0);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)  // G = dY U^T, while the first slab is staged
        umma::mma_ss(tmem, umma::desc_advance(dYk, umma::kStepK * kk), umma::desc_advance(dUk, umma::kStepK * kk), id_sq,
                     kk != 0);
      umma::commit(gbar);
    }
    __syncwarp();
  }
  const int q4 = warp & 3, h = warp >> 2;  // lane quarter of tensor memory, column part
  const int row = 32 * q4 + lane;
  const bool last_row = row == L - 1;
  const float lp_r = lp[row];
  const float es = __expf(lp[L - 1] - (last_row ? lp[0] : lp[row + 1]));
  const float2 f_r = cmulc(ph[row], ph[L - 1]);                               // f_t
  const float2 f_n = cmulc(last_row ? ph[0] : ph[row + 1], ph[L - 1]);        // f_{s+1}; f_0 for the boundary slot
  const float2 p_r = cscale(ph[row], __expf(lp_r));
  const float2 kc_r = kc[row];
  const float2 gk = cmulc(last_row ? kp[0] : cadd(cmul(mraw[row + 1], kc_r), kp[row + 1]), f_n);
  uint32_t ph_bits = 0;  // phases of the barriers
  bool ok = (umma::smem_u32(smem_raw) & 1023u) == 0;
  auto wait = [&](int which) {
    ok = umma::mbar_wait(bar0 + 8 * which, (ph_bits >> which) & 1, ok) && ok;
    ph_bits ^= 1u << which;
    __syncwarp();
  };
  const float2 zero2 = make_float2(0.f, 0.f);
  // conj(b) c;  conj(dC) c, the part through kappa against the rounded Q instead;  conj(b) xi;  and of dS'^T Q alone the
  // dots with kappa and with b
  CDot2 d_bc{zero2, zero2}, d_g = d_bc, d_x = d_bc, d_k = d_bc, d_b = d_bc;
  uint4 cr[2], br[2];                                       // raw cells of the slab

  auto slab_off = [](int r, int j) { return LONE ? umma::swz_off(r, j) : umma::swz64_off(r, j); };
  // operand tiles of slab sl
  auto stage = [&](int sl) {
    wait(3);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t off = slab_off(row, 2 * h + k);
      cr[k] = *reinterpret_cast<const uint4 *>(sC + off);
      br[k] = *reinterpret_cast<const uint4 *>(sB + off);
      const CellF cf = unpack_cell<T>(cr[k]);
      CellF bf = unpack_cell<T>(br[k]);
#pragma unroll
      for (int q = 0; q < 2; ++q) cdot2(bf.re[q], bf.im[q], cf.re[q], cf.im[q], d_bc);
      *reinterpret_cast<uint4 *>(tQ + off) = rotate_cell_split<T>(cf, f_r.x, -f_r.y);
      if (last_row) {
        const float4 *bm = reinterpret_cast<const float4 *>(bm1 + SW / 2 * sl + 8 * h + 4 * k);
        const float4 b0 = bm[0], b1 = bm[1];
        bf.re[0] = make_float2(b0.x, b0.z);
        bf.im[0] = make_float2(b0.y, b0.w);
        bf.re[1] = make_float2(b1.x, b1.z);
        bf.im[1] = make_float2(b1.y, b1.w);
      }
      *reinterpret_cast<uint4 *>(tK + off) = rotate_cell_split<T>(bf, gk.x, gk.y);
    }
    const uint32_t offz = slab_off(zp, zj);
    *reinterpret_cast<uint4 *>(tLm + offz) = split_cell(lr);
    *reinterpret_cast<uint4 *>(tZ + offz) = split_cell(zr);
    umma::fence_smem_to_async();
    umma::fence_before_sync();
  };
  // Token 127's increment path, from this thread's Lambda values (still in registers): per-warp partials of
  // (u_127 . Lambda)[d] (the warp's eight rows zp, summed over the 8 lanes that share zj) and this thread's share of
  // (k^c b_127) . Lambda[zp].
  float du127 = 0.f;
  auto helper = [&](int sl) {
    float tl[8];
    {
      const uint32_t *lw = reinterpret_cast<const uint32_t *>(&lr);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = umma::unpack2(lw[e], T());
        tl[2 * e] = v.x;
        tl[2 * e + 1] = v.y;
      }
    }
    const float4 *kbv = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(bh1) + SW * sl + 8 * zj);
    const float4 h0 = kbv[0], h1 = kbv[1];
    const float hb[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    const float uz = um[zp];
    float up[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      du127 = fmaf(hb[e], tl[e], du127);
      up[e] = uz * tl[e];
    }
    // the lanes that share zj trade halves, so that each ends with one of the eight columns (LONE: four lanes, two columns)
    const bool hi4 = lane & 4, hi8 = lane & 8, hi16 = lane & 16;
    float w4[4], w2[2];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      w4[e] = (hi16 ? up[4 + e] : up[e]) + __shfl_xor_sync(0xffffffffu, hi16 ? up[e] : up[4 + e], 16);
#pragma unroll
    for (int e = 0; e < 2; ++e)
      w2[e] = (hi8 ? w4[2 + e] : w4[e]) + __shfl_xor_sync(0xffffffffu, hi8 ? w4[e] : w4[2 + e], 8);
    const int col = 8 * zj + (hi16 ? 4 : 0) + (hi8 ? 2 : 0);
    if constexpr (LONE) {
      *reinterpret_cast<float2 *>(more + 256 + 1024 * (sl & 1) + 64 * warp + col) = make_float2(w2[0], w2[1]);
    } else {
      const float w1 = (hi4 ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, hi4 ? w2[0] : w2[1], 4);
      ulw[32 * warp + col + (hi4 ? 1 : 0)] = w1;
    }
  };

  // ---- the decay table; the first slab's operands ------------------
  if (tid < L) tab[tid] = decay_table_entry(lp, tid, L);
  stage(0);
  const bool fast_decay = !__syncthreads_or(tid < L && decay_step_out_of_range(lp, tid));
  if (warp == 1) {
    if (lane == 0 && ok && (!LONE || NB > 1)) prefetch_cb(1);  // every thread has its cells of slab 0
    __syncwarp();
  }
  helper(0);
  if (!LONE || NB > 1) prefetch_zl(1);  // (32-column slabs: at least two)
  SLX_STAMP(2);

  // ---- G -> dS' ----------------------------------------------------------
  wait(2);
  umma::fence_after_sync();
#pragma unroll 1
  for (int jj = 0; jj < PARTS; ++jj) {
    const int blk = COLS * jj + h, c0 = 32 * blk;  // blocks alternate between the warps of a row quarter
    float v[32];
    if (blk <= q4 || blk == 3) {
      umma::tmem_ld32(umma::tmem_addr(tmem, 32 * q4, c0), v);
      float g127 = v[31];
      if (blk < q4) {
        if (fast_decay) scale32(v, __expf(lp_r - lp[c0 + 1]), tab + c0);
        else decay_mask32<false>(v, c0, row, lp_r, lp, tab, 0.f);
      } else if (blk == q4) {
        float gdv = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i == lane) gdv = v[i];
        if (!last_row) gd[row] = gdv;
        if (fast_decay) decay_mask32<true>(v, c0, row, lp_r, lp, tab, 0.f);
        else decay_mask32<false>(v, c0, row, lp_r, lp, tab, 0.f);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.f;
      }
      if (blk == 3) {  // boundary slot (column 127)
        if (PREV32 && c == 0) {
#pragma unroll 1
          for (int j = 0; j < 8; ++j) {
            const uint4 y = *reinterpret_cast<const uint4 *>(tdY + umma::swz_off(row, j));
            const uint32_t *w = reinterpret_cast<const uint32_t *>(&y);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 yv = umma::unpack2(w[e], T());
              g127 = fmaf(yv.x, ulo[8 * j + 2 * e], fmaf(yv.y, ulo[8 * j + 2 * e + 1], g127));
            }
          }
        }
        v[31] = __expf(lp_r - lp[0]) * g127;
      }
    } else {  // block entirely above the diagonal
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<uint4 *>(tdS + 16384 * (blk >> 1) + umma::swz_off(row, 4 * (blk & 1) + k)) = pack8<T>(v + 8 * k);
  }
  if (warp == 0) {  // G[127][127] = dY_127 . u_127 (slot 127 of U is another token)
    const uint32_t w = *reinterpret_cast<const uint32_t *>(tdY + umma::swz_off(L - 1, lane >> 2) + 4 * (lane & 3));
    const float2 y = umma::unpack2(w, T()), u = *reinterpret_cast<const float2 *>(um + 2 * lane);
    float s = fmaf(y.x, u.x, y.y * u.y);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) gd[L - 1] = s;
  }
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  SLX_STAMP(3);
  const float gd_r = gd[row];
  const float2 cA = cscale(kc_r, gd_r);
  if (tid < L) tab[tid] = __expf(lp[tid] - lp[32 * (tid >> 5)]);  // for the tail: every reader of the first table is done
  const bool wide = ((reinterpret_cast<uintptr_t>(a.dB) | reinterpret_cast<uintptr_t>(a.dC)) & 31) == 0;
  auto store_row = [&](T *dst, const uint4 (&o)[2]) {  // 16 values of this thread's row, a whole 32-byte sector
    if (wide) {
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(o[0].x), "r"(o[0].y),
                   "r"(o[0].z), "r"(o[0].w), "r"(o[1].x), "r"(o[1].y), "r"(o[1].z), "r"(o[1].w)
                   : "memory");
    } else {
      reinterpret_cast<uint4 *>(dst)[0] = o[0];
      reinterpret_cast<uint4 *>(dst)[1] = o[1];
    }
  };
  const size_t out0 = (tok0 + row) * d.D + 16 * h;

  auto sum_ulw = [&](int sl) {  // u_127 . Lambda of a slab: sum of the per-warp partials
    if constexpr (LONE) {
      float2 acc = zero2;
#pragma unroll
      for (int w = 0; w < 16; ++w)
        acc = cadd(acc, *reinterpret_cast<const float2 *>(more + 256 + 1024 * (sl & 1) + 64 * w + 2 * lane));
      *reinterpret_cast<float2 *>(ulf + 64 * sl + 2 * lane) = acc;
    } else {
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) acc += ulw[32 * w + lane];
      ulf[32 * sl + lane] = acc;
    }
  };

  for (int sl = 0; sl < NB; ++sl) {
    SLX_STAMP(8 + 4 * sl);
    issue_first(sl);  // slab sl is staged, the accumulators of slab sl-1 are read
    if (LONE) {
      issue_second(sl);
      if (warp == 13 && sl > 0) sum_ulw(sl - 1);
    }
    if (sl > 0) {
      helper(sl);
      if (sl + 1 < NB) prefetch_zl(sl + 1);
    }
    // ---- xi = dS'^T Q + es U Lambda ------------------------------------------------------------
    wait(0);
    umma::fence_after_sync();
    SLX_STAMP(9 + 4 * sl);
    uint32_t x1[16], x2[16];  // dS'^T Q, U Lambda
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmX, 32 * q4, 16 * h), x1);
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmUL, 32 * q4, 16 * h), x2);
    umma::tmem_ld16_wait(x1);
    umma::tmem_ld16_wait(x2);
    if (!LONE) {
      umma::fence_before_sync();
      __syncthreads();  // dS'^T Q and U Lambda are in registers
      issue_second(sl);
      if (warp == 4) sum_ulw(sl);
    }
    if (last_row) {  // of the token in front of the chunk: dS'^T Q and U Lambda; token 127's own dB is formed in the tail
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = 8 * (q >> 1) + 2 * (q & 1), col = SW * sl + 16 * h + 4 * q;
        *reinterpret_cast<uint4 *>(xb + col) = make_uint4(x1[o], x1[o + 4], x1[o + 1], x1[o + 5]);
        *reinterpret_cast<uint4 *>(ub + col) = make_uint4(x2[o], x2[o + 4], x2[o + 1], x2[o + 5]);
      }
    }
    // ---- dB_s = conj(gk_s) xi_s + conj(cA_s) c_s -------------------------------------------------
    {
      uint4 o[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const CellF cf = unpack_cell<T>(cr[k]), bf = unpack_cell<T>(br[k]);
        const CellF kf = unpack_cell_split<T>(*reinterpret_cast<const uint4 *>(tK + slab_off(row, 2 * h + k)));
        uint32_t *w = reinterpret_cast<uint32_t *>(&o[k]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 x0 = tm_pair(x1 + 8 * k + 2 * q), y0 = tm_pair(x1 + 8 * k + 4 + 2 * q);
          const float2 x = __ffma2_rn(both(es), tm_pair(x2 + 8 * k + 2 * q), x0);
          const float2 y = __ffma2_rn(both(es), tm_pair(x2 + 8 * k + 4 + 2 * q), y0);
          float2 re = __fmul2_rn(both(cA.x), cf.re[q]), im = __fmul2_rn(both(cA.x), cf.im[q]);
          re = __ffma2_rn(both(cA.y), cf.im[q], re);
          im = __ffma2_rn(both(-cA.y), cf.re[q], im);
          re = __ffma2_rn(both(gk.x), x, re);
          im = __ffma2_rn(both(gk.x), y, im);
          re = __ffma2_rn(both(gk.y), y, re);
          im = __ffma2_rn(both(-gk.y), x, im);
          cdot2(bf.re[q], bf.im[q], x, y, d_x);
          cdot2(kf.re[q], kf.im[q], x0, y0, d_k);
          cdot2(bf.re[q], bf.im[q], x0, y0, d_b);
          w[2 * q] = umma::pack2(re.x, im.x, T());
          w[2 * q + 1] = umma::pack2(re.y, im.y, T());
        }
      }
      if (row < valid && !last_row) store_row(a.dB + out0 + SW * sl, o);
    }
    SLX_STAMP(10 + 4 * sl);
    // ---- dC_t = f_t (dS' kappa)_t + p_t (dY Z0)_t + cA_t b_t ------------------------------------------
    wait(1);
    umma::fence_after_sync();
    SLX_STAMP(11 + 4 * sl);
    {
      uint4 o[2];
      uint32_t t1[16], t2[16];
      umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmX2, 32 * q4, 16 * h), t1);
      umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmUL2, 32 * q4, 16 * h), t2);
      umma::tmem_ld16_wait(t1);
      umma::tmem_ld16_wait(t2);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t *r1 = t1 + 8 * k, *r2 = t2 + 8 * k;
        const CellF cf = unpack_cell<T>(cr[k]), bf = unpack_cell<T>(br[k]);
        const CellF qf = unpack_cell_split<T>(*reinterpret_cast<const uint4 *>(tQ + slab_off(row, 2 * h + k)));
        uint32_t *w = reinterpret_cast<uint32_t *>(&o[k]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 x = tm_pair(r1 + 2 * q), y = tm_pair(r1 + 4 + 2 * q);
          const float2 u = tm_pair(r2 + 2 * q), v = tm_pair(r2 + 4 + 2 * q);
          float2 re = __fmul2_rn(both(cA.x), bf.re[q]), im = __fmul2_rn(both(cA.x), bf.im[q]);
          re = __ffma2_rn(both(-cA.y), bf.im[q], re);
          im = __ffma2_rn(both(cA.y), bf.re[q], im);
          re = __ffma2_rn(both(p_r.x), u, re);
          im = __ffma2_rn(both(p_r.x), v, im);
          re = __ffma2_rn(both(-p_r.y), v, re);
          im = __ffma2_rn(both(p_r.y), u, im);
          cdot2(re, im, cf.re[q], cf.im[q], d_g);
          cdot2(x, y, qf.re[q], qf.im[q], d_g);
          re = __ffma2_rn(both(f_r.x), x, re);
          im = __ffma2_rn(both(f_r.x), y, im);
          re = __ffma2_rn(both(-f_r.y), y, re);
          im = __ffma2_rn(both(f_r.y), x, im);
          w[2 * q] = umma::pack2(re.x, im.x, T());
          w[2 * q + 1] = umma::pack2(re.y, im.y, T());
        }
      }
      if (row < valid) store_row(a.dC + out0 + SW * sl, o);
    }
    if (sl + 1 < NB) {  // every product of the slab is done: its tiles are free
      stage(sl + 1);
      __syncthreads();
    }
  }
  if (LONE) {
    __syncthreads();
    if (warp == 13) sum_ulw(NB - 1);
  }
  SLX_STAMP(4);

  // ---- fold the column halves of the per-token dots -----
  // what only the tail needs of the taps, multipliers and phases is read again, not held through the slabs
  float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row < valid) k4 = *reinterpret_cast<const float4 *>(a.K + (tok0 + row) * 4);
  const float2 kc_t = make_float2(k4.z, k4.w), k_edge = tid < 128 ? *reinterpret_cast<const float2 *>(a.K + tok0 * 4)
      : valid == L ? *reinterpret_cast<const float2 *>(a.K + (tok0 + L - 1) * 4 + 2) : zero2;  // k^p_0; k^c_127
  const float2 f_next = cmulc(last_row ? ph[0] : ph[row + 1], ph[L - 1]);
  const float lpb = last_row ? lp[0] : lp[row + 1], gd_t = gd[row];
  float2 m_own = make_float2(1.f, 0.f), m_next = m_own, zd = zero2;
  float2 c127 = zero2, b127 = zero2;  // second half: values n of token 127
  if (h == 0) {
    if (row < valid) m_own = *reinterpret_cast<const float2 *>(a.M + (tok0 + row) * 2);
    if (row + 1 < valid) m_next = *reinterpret_cast<const float2 *>(a.M + (tok0 + row + 1) * 2);
    if (last_row) zd = *reinterpret_cast<const float2 *>(a.zdot + ((size_t)bh * d.NC + c) * 2);
  } else if (h == 1 && row < d.N && valid == L) {
    c127 = load_pair<T>(a.C + (tok0 + L - 1) * d.D + 2 * row);
    b127 = load_pair<T>(a.B + (tok0 + L - 1) * d.D + 2 * row);
  }
  float2 bc = cdot2_sum(d_bc), gA = cdot2_sum(d_g), bX = cdot2_sum(d_x);
  // dM sums, over the pairs (t, s) of the chunk, differences of the same products seen from t (gA) and from s (k^c, k^p
  // against bX).  Taken with the rounded kappa and Q on both sides they cancel as the exact ones do: the term of s is
  // corrected by sum conj(kappa) X - conj(gk) sum conj(b) X, X = dS'^T Q (for the token in front of the chunk at t = 0).
  // With the unrounded b and c in these sums dM was 2.5 times as far from float64 (relative error 5e-3 against 2e-3 for one
  // chunk of N 128 in bf16).  The increment path stays with the unrounded b: its other side, <z_end, Lambda>, holds the
  // increments as the forward rounded them, and a second rounding only adds to that (a state gradient a hundred times
  // its usual size, N 64, bf16: 8.3e-3 with conj(kappa) xi, 6.8e-3 so; 1.030 and 1.050 ms for 8192 chunks of D 256).
  if (!last_row) gA = csub(gA, csub(cdot2_sum(d_k), cmul(cconj(gk), cdot2_sum(d_b))));
  bX = cmul(f_next, bX);
  pcs[L * h + row] = bc;
  if (h > 0) {
    pgs[L * (h - 1) + row] = gA;
    pbs[L * (h - 1) + row] = bX;
  }
  du127 += __shfl_xor_sync(0xffffffffu, du127, 1);
  du127 += __shfl_xor_sync(0xffffffffu, du127, 2);
  if constexpr (LONE) du127 += __shfl_xor_sync(0xffffffffu, du127, 4);
  if (zj == 0) duc[zp] = du127;
  __syncthreads();
  bc = cadd(pcs[row], pcs[L + row]);
  if constexpr (COLS == 4) bc = cadd(bc, cadd(pcs[2 * L + row], pcs[3 * L + row]));
  if (h == 0) {
#pragma unroll
    for (int k = 0; k < COLS - 1; ++k) {
      gA = cadd(gA, pgs[L * k + row]);
      bX = cadd(bX, pbs[L * k + row]);
    }
    bXs[row] = bX;
  }
  float *cB = a.carryB + ((size_t)bh * d.NC + c) * d.D;
  {
    const int n = tid & 127;  // = row
    float2 contrib = zero2, corr = zero2;
    if (n < d.N) {
      if (tid < 128) {
        // token in front of the chunk: dB_{-1}[n] = conj(k^p_0) f_0 xi[n], dk^p_0 = sum_n conj(b_{-1}[n]) f_0 xi[n]
        const float2 f_0 = cmulc(ph[0], ph[L - 1]), X = *reinterpret_cast<const float2 *>(xb + 2 * n), b = bm1[n];
        float2 ul = *reinterpret_cast<const float2 *>(ub + 2 * n);
        if (PREV32 && c == 0) {
#pragma unroll 4
          for (int p = 0; p < P; ++p) ul = cadd(ul, cscale(load_pair<T>(lam + (size_t)p * d.D + 2 * n), ulo[p]));
        }
        const float2 x = cmul(f_0, cadd(X, cscale(ul, __expf(lp[L - 1] - lp[0]))));
        *reinterpret_cast<float2 *>(cB + 2 * n) = cmul(cconj(k_edge), x);
        contrib = cmul(cconj(b), x);
        const float2 kap = cmul(cmulc(k_edge, f_0), b);
        corr = cmul(cconj(csub(umma::unpack2(umma::pack2(kap.x, kap.y, T()), T()), kap)), X);
      } else if ((tid >> 7) == 1 && valid == L) {
        // token 127: dB[n] = conj(k^c) (u_127 . Lambda)[n] + conj(k^c G) c[n]
        const float2 ul = *reinterpret_cast<const float2 *>(ulf + 2 * n);
        store_pair<T>(a.dB + (tok0 + L - 1) * d.D + 2 * n, cmul(cconj(k_edge), cadd(ul, cscale(c127, gd[L - 1]))));
        contrib = cmul(cconj(b127), ul);
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      contrib.x += __shfl_xor_sync(0xffffffffu, contrib.x, off);
      contrib.y += __shfl_xor_sync(0xffffffffu, contrib.y, off);
    }
    if (lane == 0 && warp < 8) misc[warp] = contrib;
    if (h == 0) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        corr.x += __shfl_xor_sync(0xffffffffu, corr.x, off);
        corr.y += __shfl_xor_sync(0xffffffffu, corr.y, off);
      }
      if (lane == 0) sums[4 + warp] = corr;
    }
  }
  SLX_STAMP(56);
  // ---- S^T -> S'^T (forward scores; row 127 = boundary) --------------------------------
  const float dg_r = kc_t.x * bc.x + kc_t.y * bc.y;  // Re(k^c conj(bc))
#pragma unroll 1
  for (int jj = 0; jj < PARTS; ++jj) {
    const int blk = COLS * jj + h, c0 = 32 * blk;
    float v[32];
    if (blk >= q4 || q4 == 3) {  // (the last row quarter holds the boundary row, which takes every column)
      umma::tmem_ld32(umma::tmem_addr(tmem, 32 * q4, c0), v);
      if (fast_decay) {
        scale32(v, __expf(lp[c0] - lpb), tab + c0);
        if (blk == q4 || q4 == 3) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (!last_row && c0 + i <= row) v[i] = c0 + i == row ? dg_r : 0.f;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int t = c0 + i;
          v[i] = (t > row || last_row) ? v[i] * __expf(lp[t] - lpb) : (t == row ? dg_r : 0.f);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<uint4 *>(tdS + 16384 * (blk >> 1) + umma::swz_off(row, 4 * (blk & 1) + k)) = pack8<T>(v + 8 * k);
  }
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 7) {
    if (lane == 0) {
      umma::fence_after_sync();
      constexpr uint32_t id_u = umma::make_idesc(128, 64, false, true, fmt);
      const uint64_t dSk = umma::desc_kmajor(sb + 32768, 0), dYm = umma::desc_mnmajor(sb, 0, 0);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma::mma_ss(tmem + kTmU, umma::desc_advance(dSk, 16384u * (kk >> 2) + umma::kStepK * (kk & 3)),
                     umma::desc_advance(dYm, umma::kStepMN * kk), id_u, kk != 0);
      umma::commit(gbar);
    }
    __syncwarp();
  }
  SLX_STAMP(57);
  // ---- dK and dM (under the last product): dM_t is a reverse cumulative sum over the chunk -----------------------
  float2 g_sum = zero2;
  if (h == 0) {
    const int t = row;
    float2 dkc = cscale(bc, gd_t);
    if (!last_row) dkc = cadd(dkc, cmul(cconj(m_next), bX));
    else dkc = cadd(dkc, cadd(cadd(misc[4], misc[5]), cadd(misc[6], misc[7])));
    const float2 dkp = (t == 0) ? cadd(cadd(misc[0], misc[1]), cadd(misc[2], misc[3])) : bXs[t - 1];
    if (t < valid) *reinterpret_cast<float4 *>(a.dK + (tok0 + t) * 4) = make_float4(dkp.x, dkp.y, dkc.x, dkc.y);
    float2 g = csub(gA, cadd(cmul(make_float2(k4.z, -k4.w), dkc), cmul(make_float2(k4.x, -k4.y), dkp)));
    if (t == 0) g = csub(g, cadd(cadd(sums[4], sums[5]), cadd(sums[6], sums[7])));
    if (last_row) g = cadd(g, zd);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float ox = __shfl_down_sync(0xffffffffu, g.x, off), oy = __shfl_down_sync(0xffffffffu, g.y, off);
      if (lane + off < 32) g = cadd(g, make_float2(ox, oy));
    }
    if (lane == 0) sums[warp] = g;
    g_sum = g;  // the sums of the warps above are added behind the last barrier
  }
  SLX_STAMP(58);
  wait(2);
  umma::fence_after_sync();
  SLX_STAMP(59);
  // ---- dU = increment path + score path; carry of dU ------------------------------------------
#pragma unroll 1
  for (int k2 = 0; k2 < PARTS; ++k2) {
    const int p0 = 16 * (PARTS * h + k2);
    uint32_t r0[16], r1[16];
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmR, 32 * q4, p0), r0);
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmU, 32 * q4, p0), r1);
    umma::tmem_ld16_wait(r0);
    umma::tmem_ld16_wait(r1);
    float du[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) du[i] = fmaf(es, __uint_as_float(r0[i]), __uint_as_float(r1[i]));
    if (last_row) {  // these sums belong to the token in front of the chunk
      float *cU = a.carryU + ((size_t)bh * d.NC + c) * P + p0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint4 dyr = *reinterpret_cast<const uint4 *>(tdY + umma::swz_off(L - 1, (p0 >> 3) + k));
        const uint32_t *w = reinterpret_cast<const uint32_t *>(&dyr);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 dyv = umma::unpack2(w[e], T());
          const int i = 8 * k + 2 * e;
          *reinterpret_cast<float2 *>(cU + i) = make_float2(du[i], du[i + 1]);
          du[i] = fmaf(dg_r, dyv.x, duc[p0 + i]);
          du[i + 1] = fmaf(dg_r, dyv.y, duc[p0 + i + 1]);
        }
      }
    }
    if (row < valid) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
        *reinterpret_cast<uint4 *>(a.dU + (tok0 + row) * P + p0 + 8 * k) = pack8<T>(du + 8 * k);
    }
  }
  umma::fence_before_sync();
  SLX_STAMP(5);
  const int bad = __syncthreads_or(!ok);
  if (bad) {
    if (tid == 0) umma::drain_waits(bar0, 4);
    __syncthreads();
  }
  __syncwarp();
  if (warp == 1) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, LONE ? 512 : 256);
  }
  if (!bad && h == 0 && row < valid) {
    for (int w = warp + 1; w < 4; ++w) g_sum = cadd(g_sum, sums[w]);
    const float inv = 1.f / (m_own.x * m_own.x + m_own.y * m_own.y);
    *reinterpret_cast<float2 *>(a.dM + (tok0 + row) * 2) = cscale(cmul(g_sum, m_own), inv);
  }
  if (bad) {
    // a bounded wait ran out: every gradient row of this chunk came from unfinished products or copies;
    // overwrite them (and the carries) with NaN so that the failure shows in the data as well as in the status word
    const float nanf_ = __int_as_float(0x7fc00000);
    const T nanv = from_f<T>(nanf_);
    for (int e = tid; e < valid * P; e += THREADS) a.dU[tok0 * P + e] = nanv;
    for (int e = tid; e < valid * d.D; e += THREADS) {
      a.dB[tok0 * d.D + e] = nanv;
      a.dC[tok0 * d.D + e] = nanv;
    }
    for (int e = tid; e < valid * 2; e += THREADS) a.dM[tok0 * 2 + e] = nanf_;
    for (int e = tid; e < valid * 4; e += THREADS) a.dK[tok0 * 4 + e] = nanf_;
    for (int e = tid; e < d.D; e += THREADS) cB[e] = nanf_;
    for (int e = tid; e < P; e += THREADS) a.carryU[((size_t)bh * d.NC + c) * P + e] = nanf_;
    if (tid == 0) atomicExch(&g_tc_status, 1);
  }
#undef SLX_STAMP
}

}  // namespace slx
