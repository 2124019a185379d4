// launch.h -- the kernels of the demag passes and of the Runge-Kutta stages, as
// the engine launches them.  The instantiations are compiled in one file per
// family (xpass.cu, xthree.cu, yz.cu, yzwarp.cu, yzlong.cu, yzthree.cu, thick.cu, pairs.cu), so that a change of
// one kernel compiles that family only and the families compile in parallel;
// engine.cu reaches them through these functions.  In the index-checked build
// (-DMPX_BOUNDS_CHECK) every file has its own record of the first bad index.
#pragma once
#include "../../include/mpx.h"
#include "kernels.cuh"

namespace mpx {

// ---- the pair grid of stray fields (pairfft.cuh)
// Blocks of 256 threads with 8 values each (2048 points of a transform group), 512
// where a length is 4096.
constexpr int PF_THREADS = 512;  // at most
constexpr int PF_LR = 3;         // log2 of the largest radix

struct PairFft {
  float2* t;         // work spectrum (or, while it is made, the kernel spectrum)
  const float2* ks;  // kernel spectrum
  int logP[3];
  int nin[3];   // rows of the input per axis (source grid, or the table K)
  int win[3];   // first row of the output window per axis (n_A - 1)
  int nout[3];  // rows of the output window per axis (n_B)
  float scale;  // -mu0 / (Px Py Pz)
};

// One evaluation of a pair (or the transform of its table): source and
// destination magnet slots (src -1: no gate), components, rows / columns per
// block and number of blocks of each pass.
struct PairItem {
  PairFft pf;
  int src, dst, ncomp;
  int ry_f, zc_f, tky, zc_i, ry_i;
  int g_xf, g_yf, g_z, g_yi, g_xi;
  int add;           // accumulate into out (a later source of the destination)
  const float* tab;  // the tabulated tensor (TABLE form)
  float* out;
};
// The pairs of one launch (blockIdx.y): the pairs of a world take their passes
// together, one source of every destination at a time.
constexpr int PAIR_BATCH = 8;
struct PairBatch {
  PairItem p[PAIR_BATCH];
};

using XfwdFn = void (*)(const MagnetDev*, const GroupDev*, const Work*, int, int, const float*, const float2*);
using XinvFn = void (*)(const MagnetDev*, GroupDev*, const Work*, EpiArgs, const float2*);
using LocalFn = void (*)(const MagnetDev*, GroupDev*, const Work*, EpiArgs);
using CombineFn = void (*)(const MagnetDev*, GroupDev*, const Work*, int, int);
using ControllerFn = void (*)(GroupDev*, int);
using YzFn = void (*)(const MagnetDev*, const GroupDev*, const Work*, int, int, const float2*);

// xpass.cu: everything that reads the Butcher tableau
// Forms of the x passes: warp-pair rows, rows one per warp, masked magnets, rows of
// 384 and 768 points (kernels.cuh).
struct XForm {
  bool pair = false, one = false, mask = false, three = false;
};
XfwdFn xfwd_fn(bool combine, XForm f);
XinvFn xinv_fn(XForm f);
LocalFn local_fn();
CombineFn combine_fn();
ControllerFn controller_fn();
cudaError_t upload_tableau_symbol(const TableauDev& t, cudaStream_t stream);
// xthree.cu: the forms of the x passes with `three`
XfwdFn xfwd_three_fn(bool combine, XForm f);
XinvFn xinv_three_fn(XForm f);
cudaError_t upload_tableau_three(const TableauDev& t, cudaStream_t stream);

// Launch classes of the y/z pass (yz_class of engine.cu): 0 .. 9 the block-wide
// passes (yz.cu), 10 .. 14 the warp columns of y lengths 64 .. 512 (yzwarp.cu),
// 15 .. 23 y lengths 1024 and 2048 (yzlong.cu), 24 .. 33 y lengths 96 .. 768 (yzthree.cu).
constexpr int YZ_CLASSES = 34;
YzFn yz_block_fn(int cls);
YzFn yz_warp_fn(int cls, bool one);
YzFn yz_long_fn(int cls);
YzFn yz_three_fn(int cls, bool one);

// thick.cu: the split y/z path
YzFn ycols_fn(int dir, int maxlr);
YzFn zmul_fn(int maxlr);
YzFn ycw_fn(int dir);
YzFn zcw_fn();

// Their warp-column forms (k_ycw, k_zcw of yzsplit.cuh): block sizes, columns or ky
// per block, and dynamic shared memory.
constexpr int YCW_THREADS = 256;  // 8 warps, 32 / Q columns (1024 values) each
__host__ __device__ constexpr int ycw_cols(int Py) { return (YCW_THREADS / 32) * (1024 / Py); }
__host__ __device__ constexpr int ycw_smem(int Py) {
  return ((YCW_THREADS / 32) * (1024 / Py) * qlen(Py) + Py) * (int)sizeof(float2);
}

constexpr int ZCW_UNITS = 3, ZCW_THREADS = 96 * ZCW_UNITS;
__host__ __device__ constexpr int zcw_kys(int Pz) { return ZCW_UNITS * (1024 / Pz); }
__host__ __device__ constexpr int zcw_smem(int Pz) {
  return (ZCW_UNITS * 3 * (1024 / Pz) * qlen(Pz) + Pz) * (int)sizeof(float2);
}

// pairs.cu: stray fields on the pair grid
using PairFn = void (*)(const MagnetDev*, const GroupDev*, int, int, const PairBatch, const float2*);
PairFn pair_xfwd_fn(bool table);
PairFn pair_yfft_fn(int dir);
PairFn pair_zmul_fn(bool mul);
PairFn pair_yz_fn(int logPz);
PairFn pair_xinv_fn();

#ifdef MPX_BOUNDS_CHECK
// the record of each file: read and cleared
cudaError_t bounds_take_xpass(unsigned long long* first_bad);
cudaError_t bounds_take_xthree(unsigned long long* first_bad);
cudaError_t bounds_take_yz(unsigned long long* first_bad);
cudaError_t bounds_take_yzwarp(unsigned long long* first_bad);
cudaError_t bounds_take_yzlong(unsigned long long* first_bad);
cudaError_t bounds_take_yzthree(unsigned long long* first_bad);
cudaError_t bounds_take_thick(unsigned long long* first_bad);
cudaError_t bounds_take_pairs(unsigned long long* first_bad);
#endif

}  // namespace mpx
