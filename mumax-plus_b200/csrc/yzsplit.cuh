// yzsplit.cuh -- the y/z part of the demag convolution in three passes, for
// magnets whose 3*nz columns of one kx do not fit one block (nz > 8, or long y
// transforms): the z transform then needs its own pass.
//
//   k_ycols<-1>  per group of consecutive spectrum columns (kx, c, z): load the
//                ny rows of S (zero padding above), forward FFT along y (pruned
//                first pass), store all Py rows into T[kx][c][z][ky]
//   k_zmul       per (kx, tile of ky): gather the 3 x nz values of every ky from
//                T into shared memory columns along z, forward FFT along z of
//                length Pz (pruned), 3x3 multiply by the Newell spectrum, inverse
//                FFT along z (only the nz outputs), store back into T
//   k_ycols<+1>  per group of columns: inverse FFT along y of T (only the ny
//                outputs), store into S
//
// Same arithmetic as k_yz (the same FFT passes, the same kernel spectrum
// lookup); the spectrum makes two extra round trips through global memory.
#pragma once
#include "launch.h"

namespace mpx {

// Kernel spectrum entry at (kx, ky, kz) for a runtime z length Pz, from the
// symmetry-reduced storage [kx][kz'][kcomp][ky'] (as kernel_at).
__device__ __forceinline__ void kernel_at_rt(const float* __restrict__ Kx, int kc, int hy, int kyp, float sy, int kz,
                                             int Pz, float& kxx, float& kyy, float& kzz, float& kxy, float& kxz,
                                             float& kyz, size_t left) {
  const int kzp = min(kz, Pz - kz);
  const float sz = (kz > Pz / 2) ? -1.f : 1.f;
  if (!span_ok((size_t)kzp * kc * hy + kyp + (size_t)(kc - 1) * hy, left)) {
    kxx = kyy = kzz = kxy = kxz = kyz = 0.f;
    return;
  }
  const float* Kk = Kx + (size_t)kzp * kc * hy + kyp;
  kxx = __ldg(Kk);
  kyy = __ldg(Kk + hy);
  kzz = __ldg(Kk + 2 * hy);
  kxy = sy * __ldg(Kk + 3 * hy);
  if (kc == 6) {
    kxz = sz * __ldg(Kk + 4 * hy);
    kyz = sy * sz * __ldg(Kk + 5 * hy);
  } else {
    kxz = kyz = 0.f;
  }
}

// Work item: magnet, first column (kx*3 + c)*nz + z in z, number of columns in y0.
template <int DIR, int MAXLR>
__global__ void __launch_bounds__(384, MAXLR == 3 ? 2 : 1)
    k_ycols(const MagnetDev* __restrict__ mags, const GroupDev* __restrict__ groups, const Work* __restrict__ work,
            int stage, int gate, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, gate, stage)) return;
  const int col0 = wk.z, ncol = wk.y0;
  const int ny = M.n[1];
  const int logPy = M.logP[1], Py = 1 << logPy, cs = plen(Py);
  float2* D = sm;
  float2* tws = sm + ncol * cs;
  load_twiddles<MAXLR>(tws, tw, logPy);
  float2* __restrict__ T = M.tspec + (size_t)col0 * Py;
  float2* __restrict__ S = M.spec + (size_t)col0 * ny;
  const size_t ncols_all = (size_t)M.Fh * 3 * M.n[2];  // columns of S and T (checked build)
  const size_t sleft = (ncols_all - col0) * ny, tleft = (ncols_all - col0) * Py;
  if (DIR < 0) {  // S (ny rows, zero above) -> lower half of each column
    const int logh = logPy > 0 ? logPy - 1 : 0;
    const int total = ncol << logh;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int col = e >> logh, y = e & ((1 << logh) - 1);
      D[col * cs + pidx(y)] =
          (y < ny && span_ok((size_t)col * ny + y, sleft)) ? __ldg(S + (size_t)col * ny + y) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    fft_many<-1, MAXLR, 1>(D, logPy, ncol, cs, tws);
    for (int e = threadIdx.x; e < (ncol << logPy); e += blockDim.x) {
      const int col = e >> logPy, y = e & (Py - 1);
      if (span_ok((size_t)col * Py + y, tleft)) T[(size_t)col * Py + y] = D[col * cs + pidx(y)];
    }
  } else {  // T (Py rows) -> S (the ny rows that are not padding)
    for (int e = threadIdx.x; e < (ncol << logPy); e += blockDim.x) {
      const int col = e >> logPy, y = e & (Py - 1);
      D[col * cs + pidx(y)] = span_ok((size_t)col * Py + y, tleft) ? __ldg(T + (size_t)col * Py + y)
                                                                    : make_float2(0.f, 0.f);
    }
    __syncthreads();
    fft_many<1, MAXLR, 2>(D, logPy, ncol, cs, tws);
    for (int e = threadIdx.x; e < ncol * ny; e += blockDim.x) {
      const int col = e / ny, y = e - col * ny;
      if (span_ok((size_t)col * ny + y, sleft)) S[(size_t)col * ny + y] = D[col * cs + pidx(y)];
    }
  }
}

// Work item: magnet, kx in z, first ky in y0, number of ky in ty.
template <int MAXLR>
__global__ void __launch_bounds__(384, MAXLR == 3 ? 2 : 1)
    k_zmul(const MagnetDev* __restrict__ mags, const GroupDev* __restrict__ groups, const Work* __restrict__ work,
           int stage, int gate, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, gate, stage)) return;
  const int kx = wk.z, ky0 = wk.y0, nky = wk.ty;
  const int nz = M.n[2];
  const int logPy = M.logP[1], Py = 1 << logPy;
  const int logPz = M.logP[2], Pz = 1 << logPz, cs = plen(Pz);
  const int ncol = 3 * nky;  // column (c, kyl) along z
  float2* D = sm;
  float2* tws = sm + ncol * cs;
  load_twiddles<MAXLR>(tws, tw, logPz);
  const float2* __restrict__ Tk = M.tspec + (size_t)kx * 3 * nz * Py;
  const size_t tleft = (size_t)(M.Fh - kx) * 3 * nz * Py;  // elements of T from Tk on (checked build)
  // gather: consecutive threads take consecutive ky (coalesced rows of T)
  const int logh = logPz > 0 ? logPz - 1 : 0;
  for (int e = threadIdx.x; e < (ncol << logh); e += blockDim.x) {
    const int kyl = e % nky, rest = e / nky;
    const int c = rest % 3, z = rest / 3;
    D[(c * nky + kyl) * cs + pidx(z)] = (z < nz && span_ok(((size_t)c * nz + z) * Py + ky0 + kyl, tleft))
                                            ? __ldg(Tk + ((size_t)c * nz + z) * Py + ky0 + kyl)
                                            : make_float2(0.f, 0.f);
  }
  __syncthreads();
  fft_many<-1, MAXLR, 1>(D, logPz, ncol, cs, tws);
  // 3x3 multiply by the real kernel spectrum at (kx, ky, kz)
  const int hy = Py / 2 + 1, kc = M.kcomp;
  const float* __restrict__ Kx = M.kspec + (size_t)kx * (Pz / 2 + 1) * kc * hy;
  for (int t = threadIdx.x; t < (nky << logPz); t += blockDim.x) {
    const int kyl = t % nky, kz = t / nky;
    const int ky = ky0 + kyl;
    const int kyp = min(ky, Py - ky);
    const float sy = (ky > Py / 2) ? -1.f : 1.f;
    float kxx, kyy, kzz, kxy, kxz, kyz;
    kernel_at_rt(Kx, kc, hy, kyp, sy, kz, Pz, kxx, kyy, kzz, kxy, kxz, kyz, (size_t)(M.Fh - kx) * (Pz / 2 + 1) * kc * hy);
    apply3(&D[(0 * nky + kyl) * cs + pidx(kz)], &D[(1 * nky + kyl) * cs + pidx(kz)],
           &D[(2 * nky + kyl) * cs + pidx(kz)], kxx, kyy, kzz, kxy, kxz, kyz);
  }
  __syncthreads();
  fft_many<1, MAXLR, 2>(D, logPz, ncol, cs, tws);
  float2* __restrict__ Tw = M.tspec + (size_t)kx * 3 * nz * Py;
  for (int e = threadIdx.x; e < ncol * nz; e += blockDim.x) {
    const int kyl = e % nky, rest = e / nky;
    const int c = rest % 3, z = rest / 3;
    if (span_ok(((size_t)c * nz + z) * Py + ky0 + kyl, tleft))
      Tw[((size_t)c * nz + z) * Py + ky0 + kyl] = D[(c * nky + kyl) * cs + pidx(z)];
  }
}

// --------------------------------------------------- warp columns (k_ycw, k_zcw)
// The three passes for y lengths 64 .. 1024 and z lengths 32 .. 256 in the
// four-step warp transforms of fft.cuh: a warp loads its columns straight from
// global memory, transposes once through its own shared memory and stores
// straight back, without a block barrier.  On 80 x 80 x 40 cells (padded 256 x
// 256 x 128) the block-wide passes above are bound by their barriers and
// shared-memory round trips (36 - 44 % issue active, 70.6 M warp instructions
// for k_zmul).

template <int Q, int DIR>
__device__ __forceinline__ void ycw_body(const MagnetDev& M, int col0, int ncol, float2* sm, const float2* twq) {
  constexpr int W = 32 / Q, Py = 32 * Q, cs = qlen(Py);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ny = M.n[1], first = warp * W;
  if (first >= ncol) return;
  const int nc = min(W, ncol - first);
  const size_t c0 = (size_t)col0 + first, ncols_all = (size_t)M.Fh * 3 * M.n[2];
  float2* __restrict__ S = M.spec + c0 * ny;
  float2* __restrict__ T = M.tspec + c0 * Py;
  const size_t sleft = (ncols_all - c0) * ny, tleft = (ncols_all - c0) * Py;  // checked build
  float2* C = sm + warp * W * cs;
  float2 v[32];
#pragma unroll
  for (int c = 0; c < W; ++c)
#pragma unroll
    for (int r = 0; r < Q; ++r) {
      const int y = lane + 32 * r;
      if constexpr (DIR < 0)  // S: ny rows, zero padding above (y < Py / 2 only)
        v[c * Q + r] = (c < nc && 2 * r < Q && y < ny && span_ok((size_t)c * ny + y, sleft)) ? S[(size_t)c * ny + y]
                                                                                              : make_float2(0.f, 0.f);
      else
        v[c * Q + r] = (c < nc && span_ok((size_t)c * Py + y, tleft)) ? T[(size_t)c * Py + y] : make_float2(0.f, 0.f);
    }
  four_step_inner<Q, DIR, (DIR < 0)>(v, twq, lane);
  four_step_outer<Q, DIR, (DIR > 0)>(v, C, cs, nc, lane);
  const int lc = lane / Q, ls = lane % Q;
  if (lc >= nc) return;
#pragma unroll
  for (int t = 0; t < (DIR > 0 ? 16 : 32); ++t) {  // element s + Q t of column c
    const int y = ls + Q * t;
    if constexpr (DIR < 0) {
      if (span_ok((size_t)lc * Py + y, tleft)) T[(size_t)lc * Py + y] = v[t];
    } else {
      if (y < ny && span_ok((size_t)lc * ny + y, sleft)) S[(size_t)lc * ny + y] = v[t];
    }
  }
}

// Work item as k_ycols (at most ycw_cols(Py) columns).
template <int DIR>
__global__ void __launch_bounds__(YCW_THREADS, 2)
    k_ycw(const MagnetDev* __restrict__ mags, const GroupDev* __restrict__ groups, const Work* __restrict__ work,
          int stage, int gate, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  pdl_trigger();
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, gate, stage)) {
    pdl_wait();
    return;
  }
  const int logPy = M.logP[1], Py = M.P[1];
  float2* twq = sm + (YCW_THREADS / 32) * (1024 / Py) * qlen(Py);
  if (logPy >= LOG_THREE) load_twq3(twq, tw + TW_N, Py >> 5);
  else load_twq(twq, tw, logPy);
  __syncthreads();
  pdl_wait();  // the columns are written by the previous pass
  switch (logPy) {
    case 6: ycw_body<2, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case 7: ycw_body<4, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case 8: ycw_body<8, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case 9: ycw_body<16, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case LOG_THREE: ycw_body<3, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case LOG_THREE + 1: ycw_body<6, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case LOG_THREE + 2: ycw_body<12, DIR>(M, wk.z, wk.y0, sm, twq); break;
    case LOG_THREE + 3: ycw_body<24, DIR>(M, wk.z, wk.y0, sm, twq); break;
    default: ycw_body<32, DIR>(M, wk.z, wk.y0, sm, twq); break;
  }
}

// z stage: a unit is the W = 32 / Q = 1024 / Pz consecutive ky of one kx, taken by
// three warps (one per component, W columns of length Pz = 32 Q); they meet in
// shared memory for the 3x3 multiply (a 96-thread barrier per unit).
__device__ __forceinline__ void unit_sync(int unit) { asm volatile("bar.sync %0, 96;" ::"r"(1 + unit) : "memory"); }

template <int Q>
__device__ __forceinline__ void zcw_body(const MagnetDev& M, int kx, int ky00, int nky, float2* sm,
                                         const float2* twq) {
  constexpr int W = 32 / Q, Pz = 32 * Q, cs = qlen(Pz);
  const int lane = threadIdx.x & 31, unit = threadIdx.x / 96, ut = threadIdx.x - 96 * unit, comp = ut >> 5;
  if (unit * W >= nky) return;
  const int nz = M.n[2], Py = M.P[1], ky0 = ky00 + unit * W;
  const size_t t0 = ((size_t)kx * 3 + comp) * nz * Py + ky0;
  const size_t tleft = (size_t)M.Fh * 3 * nz * Py - t0;  // checked build
  float2* __restrict__ T = M.tspec + t0;
  float2* D = sm + unit * 3 * W * cs;  // [comp][ky] columns
  float2* C = D + comp * W * cs;
  float2 v[32];
#pragma unroll
  for (int r = 0; r < Q; ++r) {  // z = lane + 32 r: W consecutive ky each, 16-byte loads
    const int z = lane + 32 * r;
    const bool in = (2 * r < Q || Q == 1) && z < nz;
#pragma unroll
    for (int c = 0; c < W; c += 2) {
      const size_t ti = (size_t)z * Py + c;
      const float4 w = (in && span_ok(ti + 1, tleft)) ? *reinterpret_cast<const float4*>(T + ti)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
      v[c * Q + r] = make_float2(w.x, w.y);
      v[(c + 1) * Q + r] = make_float2(w.z, w.w);
    }
  }
  const int lc = lane / Q, ls = lane % Q;
  four_step_inner<Q, -1, true>(v, twq, lane);
  four_step_outer<Q, -1, false>(v, C, cs, W, lane);
#pragma unroll
  for (int t = 0; t < 32; ++t) C[lc * cs + qidx(ls + Q * t)] = v[t];  // kz = s + Q t
  unit_sync(unit);
  const int hy = Py / 2 + 1, kc = M.kcomp;
  const size_t kn = (size_t)(Pz / 2 + 1) * kc * hy;
  const float* __restrict__ Kx = M.kspec + kx * kn;
  for (int t = ut; t < W * Pz; t += 96) {
    const int kyl = t % W, kz = t / W, ky = ky0 + kyl;
    const int kyp = min(ky, Py - ky);
    const float sy = (ky > Py / 2) ? -1.f : 1.f;
    float kxx, kyy, kzz, kxy, kxz, kyz;
    kernel_at<Pz>(Kx, kc, hy, kyp, sy, kz, kxx, kyy, kzz, kxy, kxz, kyz, (M.Fh - kx) * kn);
    float2* p = D + kyl * cs + qidx(kz);
    apply3(p, p + W * cs, p + 2 * W * cs, kxx, kyy, kzz, kxy, kxz, kyz);
  }
  unit_sync(unit);
#pragma unroll
  for (int c = 0; c < W; ++c)
#pragma unroll
    for (int r = 0; r < Q; ++r) v[c * Q + r] = C[c * cs + lane + 33 * r];
  four_step_inner<Q, 1, false>(v, twq, lane);
  __syncwarp();  // the columns were read by every lane
  four_step_outer<Q, 1, true>(v, C, cs, W, lane);
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    const int z = ls + Q * t;
    const size_t ti = (size_t)z * Py + lc;
    if (z < nz && span_ok(ti, tleft)) T[ti] = v[t];
  }
}

// Work item as k_zmul (at most zcw_kys(Pz) ky, a multiple of 1024 / Pz).
static __global__ void __launch_bounds__(ZCW_THREADS, 2)
    k_zcw(const MagnetDev* __restrict__ mags, const GroupDev* __restrict__ groups, const Work* __restrict__ work,
          int stage, int gate, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  pdl_trigger();
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, gate, stage)) {
    pdl_wait();
    return;
  }
  const int logPz = M.logP[2];
  float2* twq = sm + ZCW_UNITS * 3 * (1024 >> logPz) * qlen(1 << logPz);
  load_twq(twq, tw, logPz);
  __syncthreads();
  pdl_wait();  // T is written by k_ycw<-1>
  switch (logPz) {
    case 5: zcw_body<1>(M, wk.z, wk.y0, wk.ty, sm, twq); break;
    case 6: zcw_body<2>(M, wk.z, wk.y0, wk.ty, sm, twq); break;
    case 7: zcw_body<4>(M, wk.z, wk.y0, wk.ty, sm, twq); break;
    default: zcw_body<8>(M, wk.z, wk.y0, wk.ty, sm, twq); break;
  }
}

}  // namespace mpx
