// Tensor-core per-chunk backward of the v2x2ssd scan (chunk 128, P 64, half
// inputs, fp32 state).  Same mathematics as chunk_scan_bwd_kernel in
// scan_simt.cuh; every contraction runs on tcgen05 with fp32 accumulators in
// tensor memory.  One CTA of 16 worker warps and an issuing warp per (chunk, batch*head), one CTA per SM.
//
// Operands per 64-column slab of the state (half precision, every one rounded once from fp32 or as it is stored):
//   Qbar_t = c_t conj(phi_t),  kappa_s = gamma_s b_s conj(phi_{s+1}),  Bhat_s = w_s b_s,  Z0,  Lambda
// with w_s = gamma_s p_{L-1}/p_{s+1} (k^c for the last token), and per chunk
//   dS' = decay * (dY U^T),   Ye_t = exp(lp_t) dY_t,   U
//
// Tensor-memory map (fp32 columns):
//   [  0,128)  S^T = kappa Qbar^T                    (accumulated over the slabs)
//   [128,192)  dU, increment path:  Bhat Lambda^T    (accumulated over the slabs)
//   [192,448)  two buffers, one per slab parity, of  dq = dS' kappa + Ye Z0  and  X = dS'^T Qbar
//              (buffer 0 holds G = dY U^T first, and S'^T dY at the end)
//   [448,512)  UL = U Lambda of one slab
//
// The source token in front of the chunk (b_{-1}, u_{-1}) borrows key slot 127,
// whose own merged-tap column is empty (no query follows the last token):
//   dS'[t][127] = exp(lp_t - lp_0) dY_t.u_{-1},   kappa_127 = k^p_0 b_{-1} conj(phi_0)
// so that row 127 of X is the column sum the carry gradient needs, the boundary term of dq comes out of the same
// product, and row 127 of S'^T dY is the dU carried to the previous token.  What that token gets from the increment
// path, u_{-1} . Lambda and (w_{-1} b_{-1}) . Lambda, is summed on the CUDA cores (carry helpers below).
//
// What bounds it: neither HBM (35 %) nor the tensor pipe (a slab's 32 products take about 2 K cycles) but the
// rotations and the epilogue on the CUDA cores, so everything else has to run in their shadow.  The tiles of kappa,
// Qbar, Lambda and Z0 and the accumulators dq and X are double-buffered: while the tensor core works on slab i+1, all
// warps are in the epilogue of slab i and the staging of slab i+2.  Bhat and UL have one buffer, which is what shared
// and tensor memory still hold: their two products are issued behind the epilogue of the slab before and run under
// the staging of the next.  dY gives its tile to Ye and is fetched again (from L2) for the last product.  The raw
// (C, B) slab travels by TMA one slab ahead; dC / dB leave by TMA from the operand tiles.
// 8192 chunks of D 256: 1.207 ms (1.395 with single buffers, where staging, products and epilogue of a slab took
// turns).  Scaling the increment path's operands to meet the score path's (X += round(es u) round(conj(phi_{L-1})
// Lambda), dU from kappa and the same Lambda) needs neither Bhat nor UL and took 1.095 ms, but rounds two operands a
// second time: with |m| in (0.99, 1) and a large gradient of the final state dK was 2.9 times as far from float64.
//
// Thread mapping: thread = (row 32*(warp%4)+lane, 16-byte chunks 2*(warp/4) and +1 of the slab), the tensor-memory
// lane mapping, for staging and epilogue alike, so that the raw b, c of a cell stay in registers from one to the other.
#pragma once

#include "scan_tc.cuh"

namespace slx {

// tensor maps of the raw C and B operands (loads) and of dC, dB (stores): (D, T, BH), boxes of 64 columns x 128 tokens
struct alignas(64) ScanBwdMaps {
  CUtensorMap C, B, dC, dB;
};

constexpr int kTcBwdWorkers = 512, kTcBwdThreads = kTcBwdWorkers + 32;  // the last warp issues products and loads
constexpr uint32_t kBwdStage = 49152;  // [kappa 16 K][Qbar 16 K][Lambda 8 K][Z0 8 K], one per slab parity
constexpr uint32_t kBwdScalars = 81920 + 2 * kBwdStage + 32768;
constexpr size_t scan_bwd_tc_smem_bytes() { return 1024 + kBwdScalars + 17920; }
constexpr int kTmR = 128, kTmSlab = 192, kTmUL = 448, kTmU = kTmSlab;  // accumulator columns (S^T at 0)

// S^T -> S'^T of one 32-column block: row s, columns t = c0 + i.  lpb = lp_{s+1} (lp_0 for the boundary slot, whose
// row takes every column).  FAST factors exp(lp_t - lpb) through the table e3[t] = exp(lp_t - lp_{32 (t / 32)}).
template <bool FAST>
__device__ __forceinline__ void decay_mask32_rows(float (&v)[32], int c0, int s, bool boundary, float lpb,
                                                  const float *lp, const float *e3, float diag) {
  const float rf = FAST ? __expf(lp[c0] - lpb) : 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int t = c0 + i;
    const float f = FAST ? rf * e3[t] : __expf(lp[t] - lpb);
    v[i] = (t > s || boundary) ? v[i] * f : (t == s ? diag : 0.f);
  }
}

template <typename T>
__global__ void __launch_bounds__(kTcBwdThreads, 1) chunk_scan_bwd_tc_kernel(ScanBwdArgs<T> a,
                                                                              const __grid_constant__ ScanBwdMaps maps) {
  constexpr int L = kTcL, P = kTcP;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *base =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *tYe = base;                   // [t][p]  dY until G is done, then Ye
  unsigned char *tU = base + 16384;            // [s][p]
  unsigned char *tdS = base + 32768;           // 2 x [t][64 s]  dS', at the end 2 x [s][64 t]  S'^T
  unsigned char *tBh = base + 65536;           // [s][d]  Bhat
  unsigned char *tSt = base + 81920;           // two staging buffers
  unsigned char *sC = tSt + 2 * kBwdStage;     // raw C slab (swizzled tile), by TMA; dY once more at the end
  unsigned char *sB = sC + 16384;              // raw B slab
  float *lp = reinterpret_cast<float *>(base + kBwdScalars);
  float *gd = lp + L;                          // G[t][t]
  float *gm1 = gd + L;                         // dY_t . u_{-1}
  float *um1 = gm1 + L;                        // 64   u_{-1}
  float *duc = um1 + 64;                       // 64   (w_{-1} b_{-1}) . Lambda[p]
  float *e2 = duc + 64;                        // 128  decay table of dS' (decay_mask32)
  float *e3 = e2 + L;                          // 128  decay table of S'^T
  float *xb = e3 + L;                          // 256  row 127 of X, all slabs
  float *ulf = xb + 256;                       // 256  u_{-1} . Lambda, all slabs
  float *ulw = ulf + 256;                      // [16][64] per-warp partials of u_{-1} . Lambda
  float2 *gA = reinterpret_cast<float2 *>(ulw), *bX = gA + L;  // (after the slabs)
  float2 *ph = reinterpret_cast<float2 *>(ulw + 16 * 64);
  float2 *mraw = ph + L, *kc = mraw + L, *kp = kc + L, *bc = kp + L, *gsum = bc + L;
  float2 *bm1 = gsum + L;                      // 128  b_{-1}
  float2 *bh1 = bm1 + 128;                     // 128  w_{-1} b_{-1}
  float2 *misc = bh1 + 128;                    // [0] conj(b_127) . (u_127 . Lambda)   [1..4] dk^p_0, by warp   [5] zdot
  __shared__ uint64_t bars[4];  // [0], [1] products of a slab, by parity; [2] G, then S'^T dY; [3] raw slab by TMA
  __shared__ uint32_t tmem_slot;

  const ScanDims d = a.d;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool issuer = warp == kTcBwdWorkers / 32;
  auto workers_sync = [] { asm volatile("bar.sync 2, 512;" ::: "memory"); };
  const int c = blockIdx.x, bh = blockIdx.y;
  const int t0 = c * L;
  const int valid = min(L, d.T - t0);
  const size_t tok0 = (size_t)bh * d.T + t0;
  const int NB = d.D / 64;
  const uint32_t bar0 = umma::smem_u32(&bars[0]), gbar = bar0 + 16, tbar = bar0 + 24;
  constexpr int fmt = umma::HalfFmt<T>::value;

#define SLX_STAMP(i) SLX_DIAG_STAMP(i)
  SLX_STAMP(0);
  // on this path the chunk-start states are stored in the activation dtype (api: slx_scan_starts_dtype)
  const T *z0 = reinterpret_cast<const T *>(a.starts) + ((size_t)bh * d.NC + c) * P * d.D;
  const T *lam = reinterpret_cast<const T *>(a.d_inc) + ((size_t)bh * d.NC + c) * P * d.D;  // same dtype as z0
  float2 mreg[4];  // the prefix warp's multipliers, requested ahead of the bulk copies
  if (warp == 2) chunk_prefix_load4(a.M + tok0 * 2, valid, mreg);
  // U and dY land in their tiles by asynchronous copy (rows past the chunk end are zero-filled)
  auto fetch_rows = [&](unsigned char *tile, const T *src) {
    const int j = tid & 7, r0 = tid >> 3;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + 64 * i;
      const int rr = r < valid ? r : 0;
      const uint32_t nbytes = r < valid ? 16u : 0u;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(tile + umma::swz_off(r, j))),
                   "l"(src + (tok0 + rr) * P + 8 * j), "r"(nbytes)
                   : "memory");
    }
  };
  if (!issuer) {
    fetch_rows(tU, a.U);
    fetch_rows(tYe, a.dY);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // One raw (C, B) slab = two TMA boxes of [128 tokens][64 columns] into the swizzled staging tiles,
  // issued by one thread; tokens past the end of the sequence arrive as zeros.
  auto prefetch_cb = [&](int sl) {
    umma::fence_smem_to_async();  // the tiles' earlier (generic) readers are behind a barrier
    umma::mbar_expect_tx(tbar, 2u * 16384u);
    umma::tma_load_3d(umma::smem_u32(sC), &maps.C, sl * 64, t0, bh, tbar);
    umma::tma_load_3d(umma::smem_u32(sB), &maps.B, sl * 64, t0, bh, tbar);
  };
  if (tid == kTcBwdWorkers) {
#pragma unroll
    for (int i = 0; i < 4; ++i) umma::mbar_init(bar0 + 8 * i, 1);
    umma::fence_mbar_init();
    umma::tma_prefetch_map(&maps.C);
    umma::tma_prefetch_map(&maps.B);
    umma::tma_prefetch_map(&maps.dC);
    umma::tma_prefetch_map(&maps.dB);
    prefetch_cb(0);
  }
  // Z0 / Lambda slab: one 8-value (16-byte) item per thread, prefetched into registers
  const int zp = tid >> 3, zj = tid & 7;
  uint4 zr, lr;
  auto prefetch_zl = [&](int sl) {
    zr = *reinterpret_cast<const uint4 *>(z0 + (size_t)zp * d.D + sl * 64 + 8 * zj);
    lr = *reinterpret_cast<const uint4 *>(lam + (size_t)zp * d.D + sl * 64 + 8 * zj);
  };
  if (!issuer) prefetch_zl(0);

  if (issuer) {
    __syncwarp();
    umma::tmem_alloc(&tmem_slot, 512);
  }
  if (warp == 2) chunk_prefix_fast128(mreg, lp, ph, mraw, &g_scan_bad);
  if (tid >= 128 && tid < 256) {
    int t = tid - 128;
    float2 vp = make_float2(0.f, 0.f), vc = vp;
    if (t < valid) {
      float4 k4 = *reinterpret_cast<const float4 *>(a.K + (tok0 + t) * 4);
      vp = make_float2(k4.x, k4.y);
      vc = make_float2(k4.z, k4.w);
    }
    kp[t] = vp;
    kc[t] = vc;
  } else if (tid >= 256 && tid < 320) {
    int p = tid - 256;
    float v = 0.f;
    if (t0 > 0) v = to_f(a.U[(tok0 - 1) * P + p]);
    else if (a.Uprev) v = load_as_f(a.Uprev, a.prev_dtype, (size_t)bh * P + p);
    um1[p] = v;
    duc[p] = 0.f;
  } else if (tid >= 320 && tid < 320 + d.N) {
    int n = tid - 320;
    float2 bv = make_float2(0.f, 0.f);
    if (t0 > 0) bv = load_pair<T>(a.B + (tok0 - 1) * d.D + 2 * n);
    else if (a.Bprev) bv = load_as_f2(a.Bprev, a.prev_dtype, (size_t)bh * d.D + 2 * n);
    bm1[n] = bv;
  } else if (tid == 448) {
    misc[5] = *reinterpret_cast<const float2 *>(a.zdot + ((size_t)bh * d.NC + c) * 2);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");  // U, dY tiles
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t sYe = umma::smem_u32(tYe), sU = umma::smem_u32(tU), sdS = umma::smem_u32(tdS),
                 sBh = umma::smem_u32(tBh), sSt = umma::smem_u32(tSt);
  SLX_STAMP(1);
  // The products of slab sl, by one thread.  Issuing is slow (the queue in front of the tensor core is short): done by
  // a worker it held that warp, and with it every barrier, for 3 K cycles a slab; hence a warp of its own.
  constexpr uint32_t id_kk = umma::make_idesc(128, 64, false, false, fmt);
  constexpr uint32_t id_km = umma::make_idesc(128, 64, false, true, fmt);
  constexpr uint32_t id_mm = umma::make_idesc(128, 64, true, true, fmt);
  constexpr uint32_t id_sq = umma::make_idesc(128, 128, false, false, fmt);
  auto issue = [&](int sl) {  // dq, X and S^T: operands and accumulators of the slab's parity
    umma::fence_after_sync();
    const uint32_t sK = sSt + kBwdStage * (sl & 1), sQ = sK + 16384, sZ = sK + 40960;
    const uint32_t dq = tmem + kTmSlab + 128 * (sl & 1), X = dq + 64;
    const uint64_t dSk = umma::desc_kmajor(sdS, 0), dSm = umma::desc_mnmajor(sdS, 0, 16384u);
    const uint64_t dKm = umma::desc_mnmajor(sK, 0, 0), dKk = umma::desc_kmajor(sK, 0);
    const uint64_t dQm = umma::desc_mnmajor(sQ, 0, 0), dQk = umma::desc_kmajor(sQ, 0);
    const uint64_t dYk = umma::desc_kmajor(sYe, 0), dZm = umma::desc_mnmajor(sZ, 0, 0);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      umma::mma_ss(dq, umma::desc_advance(dSk, 16384u * (kk >> 2) + umma::kStepK * (kk & 3)),
                   umma::desc_advance(dKm, umma::kStepMN * kk), id_km, kk != 0);
      umma::mma_ss(X, umma::desc_advance(dSm, umma::kStepMN * kk), umma::desc_advance(dQm, umma::kStepMN * kk), id_mm,
                   kk != 0);
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      umma::mma_ss(dq, umma::desc_advance(dYk, umma::kStepK * kk), umma::desc_advance(dZm, umma::kStepMN * kk), id_km, 1);
      umma::mma_ss(tmem, umma::desc_advance(dKk, umma::kStepK * kk), umma::desc_advance(dQk, umma::kStepK * kk), id_sq,
                   (sl | kk) != 0);
    }
  };
  auto issue_increment = [&](int sl) {  // UL and the dU of the increment path, whose buffers are single
    umma::fence_after_sync();
    const uint32_t sLm = sSt + kBwdStage * (sl & 1) + 32768;
    const uint64_t dUk = umma::desc_kmajor(sU, 0), dBk = umma::desc_kmajor(sBh, 0);
    const uint64_t dLm = umma::desc_mnmajor(sLm, 0, 0), dLk = umma::desc_kmajor(sLm, 0);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      umma::mma_ss(tmem + kTmUL, umma::desc_advance(dUk, umma::kStepK * kk), umma::desc_advance(dLm, umma::kStepMN * kk),
                   id_km, kk != 0);
      umma::mma_ss(tmem + kTmR, umma::desc_advance(dBk, umma::kStepK * kk), umma::desc_advance(dLk, umma::kStepK * kk),
                   id_kk, (sl | kk) != 0);
    }
    umma::commit(bar0 + 8 * (sl & 1));  // completes with every product of the slab
  };
  if (issuer) {
    if (lane == 0) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)  // G = dY U^T, while the first slab is staged
        umma::mma_ss(tmem + kTmSlab, umma::desc_kmajor(sYe, kk), umma::desc_kmajor(sU, kk), id_sq, kk != 0);
      umma::commit(gbar);
    }
    __syncwarp();
    __syncthreads_or(0);
    // the raw tile of slab sl+1 is free once every worker has its cells of slab sl
    if (NB > 1 && lane == 0) prefetch_cb(1);
    for (int sl = 0; sl < NB; ++sl) {
      __syncthreads();  // slab sl is staged
      if (lane == 0) {
        if (sl > 0 && sl + 1 < NB) prefetch_cb(sl + 1);
        issue(sl);
      }
      __syncwarp();
      if (sl > 0) __syncthreads();  // slab sl-1 has left its accumulators, Bhat of slab sl is staged
      if (lane == 0) issue_increment(sl);
      __syncwarp();
    }
    __syncthreads();  // the last slab has left its accumulators
    __syncthreads();  // S'^T and dY are complete
    if (lane == 0) {
      umma::fence_after_sync();
      const uint32_t sdY = umma::smem_u32(sC);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma::mma_ss(tmem + kTmU, umma::desc_kmajor(sdS + 16384u * (kk >> 2), kk & 3), umma::desc_mnmajor(sdY, kk, 0),
                     id_km, kk != 0);
      umma::commit(gbar);
    }
    __syncwarp();
    __syncthreads();  // every worker has read its accumulators
    umma::tmem_dealloc(tmem, 512);
    return;
  }
  const int q4 = warp & 3, qc = warp >> 2;  // lane quarter of tensor memory, column quarter
  const int row = 32 * q4 + lane;
  const bool last_row = row == L - 1;
  const float2 ph_r = ph[row];
  const float2 kc_r = kc[row];
  // gamma_s conj(phi_{s+1}), the boundary slot: k^p_0 conj(phi_0);  w_s, the last token: k^c
  float2 gk_r = cmulc(kp[0], ph[0]), w_r = kc_r;
  if (!last_row) {
    const float2 gam = cadd(cmul(mraw[row + 1], kc_r), kp[row + 1]);
    gk_r = cmulc(gam, ph[row + 1]);
    w_r = cmul(cscale(cmulc(ph[L - 1], ph[row + 1]), __expf(lp[L - 1] - lp[row + 1])), gam);
  }
  const float lpb = last_row ? lp[0] : lp[row + 1];
  uint32_t ph_bits = 0;  // phases of the barriers: bit 0, 1 slab products, 2 gbar, 3 tbar
  bool ok = true;
  auto wait = [&](int which) {
    ok = umma::mbar_wait(bar0 + 8 * which, (ph_bits >> which) & 1) && ok;
    ph_bits ^= 1u << which;
  };
  float2 acc_bc = make_float2(0.f, 0.f);  // conj(b) c over this thread's cells
  uint4 cr[2], br[2], cn[2], bn[2];       // raw cells: slab in its epilogue, slab being staged

  // Operand tiles of slab sl from its raw cells, written to its staging buffer.  The bulk stores of dC / dB of
  // slab sl-2 leave from the same tiles: the rotated cells wait in registers until those have read them.
  auto stage = [&](int sl) {
    wait(3);
    uint4 qv[2], kv[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t off = umma::swz_off(row, 2 * qc + k);
      cn[k] = *reinterpret_cast<const uint4 *>(sC + off);
      bn[k] = *reinterpret_cast<const uint4 *>(sB + off);
      uint4 src = bn[k];
      if (last_row) {
        float tmp[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = bm1[sl * 32 + 8 * qc + 4 * k + e];
          tmp[2 * e] = v.x;
          tmp[2 * e + 1] = v.y;
        }
        src = pack8<T>(tmp);
      }
      qv[k] = rotate_chunk<T>(cn[k], cconj(ph_r));
      kv[k] = rotate_chunk<T>(src, gk_r);
      cdot_chunk<T>(bn[k], cn[k], acc_bc);
    }
    unsigned char *buf = tSt + kBwdStage * (sl & 1);
    if (sl >= 2) {
      if (tid == 0) umma::tma_store_wait_read();
      workers_sync();
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t off = umma::swz_off(row, 2 * qc + k);
      *reinterpret_cast<uint4 *>(buf + off) = kv[k];
      *reinterpret_cast<uint4 *>(buf + 16384 + off) = qv[k];
    }
    *reinterpret_cast<uint4 *>(buf + 32768 + umma::swz_off(zp, zj)) = lr;
    *reinterpret_cast<uint4 *>(buf + 40960 + umma::swz_off(zp, zj)) = zr;
    umma::fence_smem_to_async();
    umma::fence_before_sync();
  };
  // Bhat of the slab just staged, from the raw cells in registers
  auto stage_bhat = [&]() {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      *reinterpret_cast<uint4 *>(tBh + umma::swz_off(row, 2 * qc + k)) = rotate_chunk<T>(bn[k], w_r);
  };
  // The increment path of the token in front of the chunk, from this thread's Lambda values (still in registers):
  // per-warp partials of (u_{-1} . Lambda)[d] (rows zp of this warp, summed over the 4 lanes that share zj) and
  // duc[p] += sum_d bh1[d] Lambda[p][d] (summed over the 8 lanes that share zp).
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
    const float4 *kbv = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(bh1) + 64 * sl + 8 * zj);
    const float4 h0 = kbv[0], h1 = kbv[1];
    const float hb[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    const float uz = um1[zp];
    float ds = 0.f, up[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      ds = fmaf(hb[e], tl[e], ds);
      up[e] = uz * tl[e];
    }
    // sums over the four lanes that share zj: the lanes trade halves, so that each ends with two of the eight columns
    const bool hi8 = lane & 8, hi16 = lane & 16;
    float w4[4], w2[2];
#pragma unroll
    for (int e = 0; e < 4; ++e) w4[e] = (hi8 ? up[4 + e] : up[e]) + __shfl_xor_sync(0xffffffffu, hi8 ? up[e] : up[4 + e], 8);
#pragma unroll
    for (int e = 0; e < 2; ++e) w2[e] = (hi16 ? w4[2 + e] : w4[e]) + __shfl_xor_sync(0xffffffffu, hi16 ? w4[e] : w4[2 + e], 16);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) ds += __shfl_xor_sync(0xffffffffu, ds, off);
    if (zj == 0) duc[zp] += ds;
    *reinterpret_cast<float2 *>(ulw + 64 * warp + 8 * zj + (hi8 ? 4 : 0) + (hi16 ? 2 : 0)) = make_float2(w2[0], w2[1]);
  };

  // ---- the boundary dots, the decay tables; the first slab's operands ------------------
  {
    const int j = tid & 7, r0 = tid >> 3;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + 64 * i;
      const uint4 dyr = *reinterpret_cast<const uint4 *>(tYe + umma::swz_off(r, j));
      const uint32_t *w = reinterpret_cast<const uint32_t *>(&dyr);
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = umma::unpack2(w[e], T());
        dot = fmaf(v.x, um1[8 * j + 2 * e], fmaf(v.y, um1[8 * j + 2 * e + 1], dot));
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (j == 0) gm1[r] = dot;
    }
  }
  if (tid < L) {
    e2[tid] = decay_table_entry(lp, tid, L);
    e3[tid] = __expf(lp[tid] - lp[32 * (tid >> 5)]);
  } else if (tid >= 256 && tid < 256 + d.N) {
    const float2 s0 = cscale(cmulc(ph[L - 1], ph[0]), __expf(lp[L - 1] - lp[0]));  // p_{L-1}/p_0
    bh1[tid - 256] = cmul(cmul(s0, kp[0]), bm1[tid - 256]);
  }
  stage(0);
  stage_bhat();
  umma::fence_smem_to_async();
  const bool fast_decay = !__syncthreads_or(tid < L && decay_step_out_of_range(lp, tid));
  helper(0);
  if (NB > 1) prefetch_zl(1);
  SLX_STAMP(2);

  // ---- G -> dS'; dY -> Ye in its place ----------------------------------------------------------
  wait(2);
  umma::fence_after_sync();
  {
    const int j = tid & 7, r0 = tid >> 3;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + 64 * i;
      uint4 *cell = reinterpret_cast<uint4 *>(tYe + umma::swz_off(r, j));
      const uint4 dyr = *cell;
      const uint32_t *w = reinterpret_cast<const uint32_t *>(&dyr);
      const float el = __expf(lp[r]);
      float ty[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = umma::unpack2(w[e], T());
        ty[2 * e] = el * v.x;
        ty[2 * e + 1] = el * v.y;
      }
      *cell = pack8<T>(ty);
    }
  }
  {
    const float lpt = lp[row];
    const int c0 = 32 * qc;
    float v[32];
    if (qc <= q4) {
      umma::tmem_ld32(umma::tmem_addr(tmem + kTmSlab, 32 * q4, c0), v);
      if (qc == q4) {  // the diagonal lives in the block with qc == q4
        float gdv = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i == lane) gdv = v[i];
        gd[row] = gdv;
      }
      if (fast_decay) decay_mask32<true>(v, c0, row, lpt, lp, e2, 0.f);
      else decay_mask32<false>(v, c0, row, lpt, lp, e2, 0.f);
    } else {  // block entirely above the diagonal
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
    if (qc == 3) v[31] = __expf(lpt - lp[0]) * gm1[row];  // boundary slot (column 127)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<uint4 *>(tdS + 16384 * (qc >> 1) + umma::swz_off(row, 4 * (qc & 1) + k)) = pack8<T>(v + 8 * k);
  }
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  SLX_STAMP(3);
  const float gd_r = gd[row];
  const float2 cA_r = cscale(kc_r, gd_r);

  float2 pgA = make_float2(0.f, 0.f), pX = pgA, pUL = pgA;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    cr[k] = cn[k];
    br[k] = bn[k];
  }
  for (int sl = 0; sl < NB; ++sl) {
    SLX_STAMP(8 + 8 * sl);
    // u_{-1} . Lambda of this slab: sum of the 16 per-warp partials (two warps, one column per thread)
    if (tid >= 32 && tid < 96) {
      const int dcol = tid - 32;
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 16; ++w) acc += ulw[64 * w + dcol];
      ulf[64 * sl + dcol] = acc;
    }
    if (sl + 1 < NB) {
      stage(sl + 1);
      SLX_STAMP(9 + 8 * sl);
      __syncthreads();
      SLX_STAMP(10 + 8 * sl);
      helper(sl + 1);
      if (sl + 2 < NB) prefetch_zl(sl + 2);
    } else {
      // the raw tiles are free: dY comes back for the last product
      fetch_rows(sC, a.dY);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    SLX_STAMP(11 + 8 * sl);
    wait(sl & 1);
    umma::fence_after_sync();
    SLX_STAMP(12 + 8 * sl);
    // ---- slab epilogue: dC, dB, per-token dots --------------------------------------------------
    //   dC_t = phi_t dq_t + (k^c_t G_tt) b_t,
    //   dB_s = (conj(k^c_s) G_ss) c_s + conj(gk_s) X_s + conj(w_s) UL_s
    //   dots: gA += c conj(dC),  conj(b) X,  conj(b) UL
    // Row 127 of X belongs to the token in front of the chunk; the last token takes no part in X.
    unsigned char *buf = tSt + kBwdStage * (sl & 1);
    const uint32_t acc = tmem + kTmSlab + 128 * (sl & 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      // eight accumulator columns (four complex lanes) of dq, X and UL at a time
      uint32_t r0[8], r1[8], r2[8];
      umma::tmem_ld8_issue(umma::tmem_addr(acc, 32 * q4, 16 * qc + 8 * k), r0);
      umma::tmem_ld8_issue(umma::tmem_addr(acc, 32 * q4, 64 + 16 * qc + 8 * k), r1);
      umma::tmem_ld8_issue(umma::tmem_addr(tmem + kTmUL, 32 * q4, 16 * qc + 8 * k), r2);
      umma::tmem_ld8_wait(r0);
      umma::tmem_ld8_wait(r1);
      umma::tmem_ld8_wait(r2);
      if (last_row) {
        float4 *dst = reinterpret_cast<float4 *>(xb + 64 * sl + 16 * qc + 8 * k);
#pragma unroll
        for (int i = 0; i < 2; ++i)
          dst[i] = make_float4(__uint_as_float(r1[4 * i]), __uint_as_float(r1[4 * i + 1]),
                               __uint_as_float(r1[4 * i + 2]), __uint_as_float(r1[4 * i + 3]));
#pragma unroll
        for (int i = 0; i < 8; ++i) r1[i] = 0;
      }
      const uint32_t *wb = reinterpret_cast<const uint32_t *>(&br[k]);
      const uint32_t *wc = reinterpret_cast<const uint32_t *>(&cr[k]);
      float odc[8], odb[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 bv = umma::unpack2(wb[e], T()), cv = umma::unpack2(wc[e], T());
        const float2 dqv = make_float2(__uint_as_float(r0[2 * e]), __uint_as_float(r0[2 * e + 1]));
        const float2 Xv = make_float2(__uint_as_float(r1[2 * e]), __uint_as_float(r1[2 * e + 1]));
        const float2 ULv = make_float2(__uint_as_float(r2[2 * e]), __uint_as_float(r2[2 * e + 1]));
        const float2 dcv = cmadd(ph_r, dqv, cmul(cA_r, bv));
        pgA = cmadd(cv, cconj(dcv), pgA);
        const float2 dbv = cmadd(cconj(gk_r), Xv, cmadd(cconj(w_r), ULv, cmul(cconj(cA_r), cv)));
        pX = cmadd(cconj(bv), Xv, pX);
        pUL = cmadd(cconj(bv), ULv, pUL);
        odc[2 * e] = dcv.x;
        odc[2 * e + 1] = dcv.y;
        odb[2 * e] = dbv.x;
        odb[2 * e + 1] = dbv.y;
      }
      // the results take the place of the slab's (now idle) Qbar / kappa cells and leave from there
      const uint32_t off = umma::swz_off(row, 2 * qc + k);
      *reinterpret_cast<uint4 *>(buf + 16384 + off) = pack8<T>(odc);
      *reinterpret_cast<uint4 *>(buf + off) = pack8<T>(odb);
    }
    if (sl + 1 < NB) stage_bhat();  // of slab sl+1: the product that read the last one is done
    umma::fence_smem_to_async();  // Bhat, and the dC / dB cells, which leave through the async proxy
    umma::fence_before_sync();
    SLX_STAMP(13 + 8 * sl);
    __syncthreads();
    SLX_STAMP(14 + 8 * sl);
    if (tid == 0) {  // one thread sends both tiles (rows past the end of the sequence are clipped by the copy)
      umma::tma_store_3d(&maps.dC, 64 * sl, t0, bh, sSt + kBwdStage * (sl & 1) + 16384);
      umma::tma_store_3d(&maps.dB, 64 * sl, t0, bh, sSt + kBwdStage * (sl & 1));
      umma::tma_store_commit();
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      cr[k] = cn[k];
      br[k] = bn[k];
    }
  }
  SLX_STAMP(4);

  // ---- fold the column quarters of the per-token dots (scratch: the idle Lambda and Z0 tiles) -----
  float2 *part = reinterpret_cast<float2 *>(tSt + 32768);  // 3 x [4][128]: gA, bX, bc
  part[128 * qc + row] = pgA;
  // conj(b_s) xi_s = phi_{s+1} conj(b) X + conj(p_{L-1}/p_{s+1}) conj(b) UL; row 127: conj(b_127) . (u_127 . Lambda)
  if (!last_row) {
    const float2 sg = cscale(cmulc(ph[L - 1], ph[row + 1]), __expf(lp[L - 1] - lp[row + 1]));
    pUL = cmadd(ph[row + 1], pX, cmul(cconj(sg), pUL));
  }
  part[512 + 128 * qc + row] = pUL;
  part[1024 + 128 * qc + row] = acc_bc;
  workers_sync();
  {
    // every thread needs its row's bc (diagonal of S'^T); the first quarter keeps the sums for the token phase
    const float2 s2 = cadd(cadd(part[1024 + row], part[1152 + row]), cadd(part[1280 + row], part[1408 + row]));
    acc_bc = s2;
    if (qc == 0) {
      gA[row] = cadd(cadd(part[row], part[128 + row]), cadd(part[256 + row], part[384 + row]));
      const float2 s1 = cadd(cadd(part[512 + row], part[640 + row]), cadd(part[768 + row], part[896 + row]));
      bX[row] = s1;
      if (last_row) misc[0] = s1;
      bc[row] = s2;
    }
  }
  // Gradient of the token before the chunk: xi_n = phi_0 X_127[n] + conj(p_{L-1}/p_0) (u_{-1} . Lambda)[n],
  // dB_{-1}[n] = conj(k^p_0) xi_n, dk^p_0 = sum_n conj(b_{-1}[n]) xi_n
  float *cB = a.carryB + ((size_t)bh * d.NC + c) * d.D;
  if (tid >= 256 && tid < 256 + L) {
    const int n = tid - 256;
    float2 contrib = make_float2(0.f, 0.f);
    if (n < d.N) {
      const float2 s0 = cscale(cmulc(ph[L - 1], ph[0]), __expf(lp[L - 1] - lp[0]));
      const float2 xi = cmadd(ph[0], make_float2(xb[2 * n], xb[2 * n + 1]),
                              cmul(cconj(s0), make_float2(ulf[2 * n], ulf[2 * n + 1])));
      *reinterpret_cast<float2 *>(cB + 2 * n) = cmul(cconj(kp[0]), xi);
      contrib = cmul(cconj(bm1[n]), xi);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      contrib.x += __shfl_xor_sync(0xffffffffu, contrib.x, off);
      contrib.y += __shfl_xor_sync(0xffffffffu, contrib.y, off);
    }
    if (lane == 0) misc[1 + warp - 8] = contrib;
  }
  SLX_STAMP(56);
  // ---- S^T -> S'^T (forward scores; row 127 = boundary) --------------------------------
  const float dg_r = kc_r.x * acc_bc.x + kc_r.y * acc_bc.y;  // Re(k^c conj(bc))
  {
    const int c0 = 32 * qc;
    float v[32];
    if (qc >= q4 || q4 == 3) {  // (the last row quarter holds the boundary row, which takes every column)
      umma::tmem_ld32(umma::tmem_addr(tmem, 32 * q4, c0), v);
      if (fast_decay) decay_mask32_rows<true>(v, c0, row, last_row, lpb, lp, e3, dg_r);
      else decay_mask32_rows<false>(v, c0, row, last_row, lpb, lp, e3, dg_r);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<uint4 *>(tdS + 16384 * (qc >> 1) + umma::swz_off(row, 4 * (qc & 1) + k)) = pack8<T>(v + 8 * k);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");  // dY
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  SLX_STAMP(57);
  // ---- dK and the per-token terms of dM (overlaps the last product) -----------------------
  if (tid < L) {
    const int t = tid;
    float2 dkc = cscale(bc[t], gd[t]);
    if (t + 1 < L) dkc = cadd(dkc, cmul(cconj(mraw[t + 1]), bX[t]));
    else dkc = cadd(dkc, misc[0]);
    const float2 dkp = (t == 0) ? cadd(cadd(misc[1], misc[2]), cadd(misc[3], misc[4])) : bX[t - 1];
    if (t < valid) *reinterpret_cast<float4 *>(a.dK + (tok0 + t) * 4) = make_float4(dkp.x, dkp.y, dkc.x, dkc.y);
    float2 g = csub(gA[t], cadd(cmul(cconj(kc[t]), dkc), cmul(cconj(kp[t]), dkp)));
    if (t == L - 1) {
      g = cadd(g, misc[5]);
    }
    gsum[t] = g;
    asm volatile("bar.sync 1, 128;" ::: "memory");  // gsum of the four token warps is complete
  }
  // reverse cumulative sum of g over the chunk (warp 0: 4 tokens per lane + shuffle scan)
  if (warp == 0) {
    float2 loc[4];
    float2 run = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 3; i >= 0; --i) {
      run = cadd(run, gsum[4 * lane + i]);
      loc[i] = run;
    }
    float2 incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      float ox = __shfl_down_sync(0xffffffffu, incl.x, off), oy = __shfl_down_sync(0xffffffffu, incl.y, off);
      if (lane + off < 32) incl = cadd(incl, make_float2(ox, oy));
    }
    const float2 excl = csub(incl, run);  // sum over the lanes above
#pragma unroll
    for (int i = 0; i < 4; ++i) gsum[4 * lane + i] = cadd(loc[i], excl);
  }
  SLX_STAMP(58);
  wait(2);
  umma::fence_after_sync();
  SLX_STAMP(59);
  // ---- dU = increment path + score path; carry of dU ------------------------------------------
  {
    uint32_t r0[16], r1[16];
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmR, 32 * q4, 16 * qc), r0);
    umma::tmem_ld16_issue(umma::tmem_addr(tmem + kTmU, 32 * q4, 16 * qc), r1);
    umma::tmem_ld16_wait(r0);
    umma::tmem_ld16_wait(r1);
    float du[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) du[i] = __uint_as_float(r0[i]);
    if (last_row) {  // the score path's sum belongs to the token in front of the chunk
      float *cU = a.carryU + ((size_t)bh * d.NC + c) * P + 16 * qc;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint4 dyr = *reinterpret_cast<const uint4 *>(sC + umma::swz_off(L - 1, 2 * qc + k));
        const uint32_t *w = reinterpret_cast<const uint32_t *>(&dyr);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 dyv = umma::unpack2(w[e], T());
          const int i = 8 * k + 2 * e;
          cU[i] = __uint_as_float(r1[i]) + duc[16 * qc + i];
          cU[i + 1] = __uint_as_float(r1[i + 1]) + duc[16 * qc + i + 1];
          du[i] = fmaf(dg_r, dyv.x, du[i]);
          du[i + 1] = fmaf(dg_r, dyv.y, du[i + 1]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) du[i] += __uint_as_float(r1[i]);
    }
    if (row < valid) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
        *reinterpret_cast<uint4 *>(a.dU + (tok0 + row) * P + 16 * qc + 8 * k) = pack8<T>(du + 8 * k);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (tid < valid) {
    const float2 m = mraw[tid];
    const float inv = 1.f / (m.x * m.x + m.y * m.y);
    *reinterpret_cast<float2 *>(a.dM + (tok0 + tid) * 2) = cscale(cmul(gsum[tid], m), inv);
  }
  SLX_STAMP(5);
  if (tid == 0) umma::tma_store_wait_all();  // the bulk stores of dC / dB have completed
  int bad;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 2, 512, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(bad)
      : "r"(ok ? 0 : 1)
      : "memory");
  if (bad) {
    // a bounded wait ran out: every gradient row of this chunk came from unfinished products or copies;
    // overwrite them (and the carries) with NaN so that the failure shows in the data as well as in the status word
    const float nanf_ = __int_as_float(0x7fc00000);
    const T nanv = from_f<T>(nanf_);
    for (int e = tid; e < valid * P; e += kTcBwdWorkers) a.dU[tok0 * P + e] = nanv;
    for (int e = tid; e < valid * d.D; e += kTcBwdWorkers) {
      a.dB[tok0 * d.D + e] = nanv;
      a.dC[tok0 * d.D + e] = nanv;
    }
    for (int e = tid; e < valid * 2; e += kTcBwdWorkers) a.dM[tok0 * 2 + e] = nanf_;
    for (int e = tid; e < valid * 4; e += kTcBwdWorkers) a.dK[tok0 * 4 + e] = nanf_;
    for (int e = tid; e < d.D; e += kTcBwdWorkers) cB[e] = nanf_;
    for (int e = tid; e < P; e += kTcBwdWorkers) a.carryU[((size_t)bh * d.NC + c) * P + e] = nanf_;
    if (tid == 0) atomicExch(&g_tc_status, 1);
  }
#undef SLX_STAMP
}

}  // namespace slx
