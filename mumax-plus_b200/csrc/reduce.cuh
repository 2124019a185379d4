// reduce.cuh -- reductions, samples, state initialisation and the minimizer's
// kernels.  Included by engine.cu only.
#pragma once
#include "kernels.cuh"

namespace mpx {

// ---------------------------------------------------------------- reductions
// Deterministic two-level reductions over the geometry: block partials in a
// fixed order, then one block.  op 0: per-component sum, op 1: max |v|.
static __global__ void k_reduce_partial(const float* __restrict__ a, int N, int ncomp,
                                 const unsigned char* __restrict__ geom, int op, double* partial) {
  __shared__ double sh[3][256];
  double acc[3] = {0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    if (geom && !geom[i]) continue;
    if (op == 0) {
      for (int c = 0; c < ncomp; ++c) acc[c] += (double)a[(size_t)c * N + i];
    } else if (op == 2) {  // sum of squared norms (dotSum(a, a), core/reduce.cu)
      for (int c = 0; c < ncomp; ++c) {
        const double v = a[(size_t)c * N + i];
        acc[0] += v * v;
      }
    } else {
      double s = 0;
      for (int c = 0; c < ncomp; ++c) {
        const double v = a[(size_t)c * N + i];
        s += v * v;
      }
      s = sqrt(s);
      acc[0] = (s > acc[0] || s != s) ? s : acc[0];
    }
  }
  for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int c = 0; c < 3; ++c) {
        if (op != 1) sh[c][threadIdx.x] += sh[c][threadIdx.x + s];
        else {
          const double o = sh[c][threadIdx.x + s];
          if (o > sh[c][threadIdx.x] || o != o) sh[c][threadIdx.x] = o;
        }
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; ++c) partial[blockIdx.x * 3 + c] = sh[c][0];
}

// The block partials are added in block order by one thread per component;
// staging them in shared memory first takes the serial chain from a global load
// per term (27 us for 256 blocks) to an FP64 add per term.
constexpr int REDUCE_MAX_BLOCKS = 256;
static __global__ void __launch_bounds__(256) k_reduce_final(const double* __restrict__ partial, int nblocks, int op,
                                                             double* out) {
  __shared__ double sp[3 * REDUCE_MAX_BLOCKS];
  for (int i = threadIdx.x; i < 3 * nblocks; i += blockDim.x) sp[i] = partial[i];
  __syncthreads();
  if (threadIdx.x >= 3) return;
  double r = 0;
  for (int b = 0; b < nblocks; ++b) {
    const double v = sp[b * 3 + threadIdx.x];
    if (op != 1) r += v;
    else if (v > r || v != v) r = v;
  }
  out[threadIdx.x] = r;
}

// Sampled run: <m> of one magnet into the due rows of its group's table, with
// the arithmetic of mpx_average (k_reduce_partial / k_reduce_final over the
// same 256 x 256 grid), so the values equal a host-side average of the state.
// Both kernels do nothing unless rows are due.
static __global__ void __launch_bounds__(256) k_sample_partial(const MagnetDev* __restrict__ mags,
                                                        const GroupDev* __restrict__ groups, int slot,
                                                        double* partial) {
  __shared__ double sh[3][256];
  const MagnetDev& M = mags[slot];
  const GroupDev& G = groups[M.group];
  if (G.samp_hi <= G.samp_lo) return;
  const int N = M.N;
  const float* __restrict__ a = M.buf[G.map[0]];
  const unsigned char* __restrict__ geom = M.geom;
  double acc[3] = {0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    if (geom && !geom[i]) continue;
    for (int c = 0; c < 3; ++c) acc[c] += (double)a[(size_t)c * N + i];
  }
  for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] += sh[c][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; ++c) partial[blockIdx.x * 3 + c] = sh[c][0];
}

static __global__ void __launch_bounds__(256) k_sample_final(const MagnetDev* __restrict__ mags,
                                                             const GroupDev* __restrict__ groups, int slot,
                                                             const double* __restrict__ partial, int nblocks,
                                                             long long ngeo, int col) {
  __shared__ double sp[3 * REDUCE_MAX_BLOCKS];
  const GroupDev& G = groups[mags[slot].group];
  if (G.samp_hi <= G.samp_lo) return;
  for (int i = threadIdx.x; i < 3 * nblocks; i += blockDim.x) sp[i] = partial[i];
  __syncthreads();
  if (threadIdx.x >= 3) return;
  double r = 0;
  for (int b = 0; b < nblocks; ++b) r += sp[b * 3 + threadIdx.x];
  for (int row = G.samp_lo; row < G.samp_hi; ++row)
    G.samp_out[(size_t)row * G.samp_row + col + threadIdx.x] = ngeo > 0 ? r / ngeo : 0.0;
}

// Set m: normalise per cell inside the geometry (core/variable.cpp:76-87).
static __global__ void k_normalize_into(float* dst, const float* __restrict__ src, int N,
                                 const unsigned char* __restrict__ geom) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  float x = src[i], y = src[N + i], z = src[2 * N + i];
  if (!geom || geom[i]) {
    const float inv = rsqrtf(x * x + y * y + z * z);
    x *= inv;
    y *= inv;
    z *= inv;
  }
  dst[i] = x;
  dst[N + i] = y;
  dst[2 * N + i] = z;
}

// n normal(0,1) numbers for the initial magnetisation of a new magnet: the
// splitmix64 finaliser of (seed, index) (Steele, Lea and Flood, OOPSLA 2014)
// gives two 24-bit uniforms, turned into one normal by Box-Muller.
static __global__ void k_random_normal(float* __restrict__ out, int n, unsigned long long seed) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const float u1 = (float)((unsigned)(z >> 40) + 1u) * (1.0f / 16777216.0f);  // (0, 1]
    const float u2 = (float)(unsigned)(z & 0xFFFFFFull) * (1.0f / 16777216.0f);  // [0, 1)
    out[i] = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
  }
}

// ------------------------------------------------------------- minimizer
// One steepest-descent step of physics/minimizer.cu (k_step): from the state m0
// and its damping torque t0, m1 = ((4 - dt^2 t0^2) m0 + 4 dt t0) / (4 + dt^2 t0^2)
// over every cell of the grid; m0 and the unnormalised m1 are kept for the
// Barzilai-Borwein step size, the state becomes m1 normalised inside the
// geometry (the reference's magnetization()->set(m1)).
static __global__ void k_min_step(float* __restrict__ state, float* __restrict__ m0_out, float* __restrict__ m1_out,
                           const float* __restrict__ t0, int N, float dt, const unsigned char* __restrict__ geom) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const float3 m0 = load3(state, N, i), t = load3(t0, N, i);
    const float t2 = dt * dt * dot3(t, t);
    const float inv = 1.0f / (4.0f + t2);
    const float3 m1 = f3(((4.0f - t2) * m0.x + 4.0f * dt * t.x) * inv, ((4.0f - t2) * m0.y + 4.0f * dt * t.y) * inv,
                         ((4.0f - t2) * m0.z + 4.0f * dt * t.z) * inv);
    store3(m0_out, N, i, m0);
    store3(m1_out, N, i, m1);
    float3 n = m1;
    if (!geom || geom[i]) {
      const float r = rsqrtf(dot3(m1, m1));
      n = f3(m1.x * r, m1.y * r, m1.z * r);
    }
    store3(state, N, i, n);
  }
}

// Block partials (FP64) of dm.dm, dm.dt, dt.dt and max|dm| with dm = m1 - m0 and
// dt = t0 - t1 (physics/minimizer.cu: BarzilianBorweinStepSize, maxVecNorm(dm)).
static __global__ void k_min_partial(const float* __restrict__ m0, const float* __restrict__ m1, const float* __restrict__ t0,
                              const float* __restrict__ t1, int N, double* __restrict__ partial) {
  __shared__ double sh[4][256];
  double a = 0, b = 0, c = 0, mx = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const float3 p = load3(m0, N, i), q = load3(m1, N, i), u = load3(t0, N, i), v = load3(t1, N, i);
    const float3 dm = f3(q.x - p.x, q.y - p.y, q.z - p.z);
    const float3 dt = f3(u.x - v.x, u.y - v.y, u.z - v.z);
    const double mm = (double)dm.x * dm.x + (double)dm.y * dm.y + (double)dm.z * dm.z;
    a += mm;
    b += (double)dm.x * dt.x + (double)dm.y * dt.y + (double)dm.z * dt.z;
    c += (double)dt.x * dt.x + (double)dt.y * dt.y + (double)dt.z * dt.z;
    const double n = sqrt(mm);
    mx = (n > mx || n != n) ? n : mx;
  }
  sh[0][threadIdx.x] = a;
  sh[1][threadIdx.x] = b;
  sh[2][threadIdx.x] = c;
  sh[3][threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      for (int k = 0; k < 3; ++k) sh[k][threadIdx.x] += sh[k][threadIdx.x + s];
      const double o = sh[3][threadIdx.x + s];
      if (o > sh[3][threadIdx.x] || o != o) sh[3][threadIdx.x] = o;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; ++k) partial[blockIdx.x * 4 + k] = sh[k][0];
}

static __global__ void __launch_bounds__(256) k_min_final(const double* __restrict__ partial, int nblocks,
                                                          double* __restrict__ out) {
  __shared__ double sp[4 * REDUCE_MAX_BLOCKS];
  for (int i = threadIdx.x; i < 4 * nblocks; i += blockDim.x) sp[i] = partial[i];
  __syncthreads();
  if (threadIdx.x >= 4) return;
  double r = 0;
  for (int b = 0; b < nblocks; ++b) {
    const double v = sp[b * 4 + threadIdx.x];
    if (threadIdx.x < 3) r += v;
    else if (v > r || v != v) r = v;
  }
  out[threadIdx.x] = r;
}

}  // namespace mpx
