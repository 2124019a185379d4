// newell.cuh -- FP64 construction of the demag kernel and its spectrum.
//
// The Newell tensor (Newell, Williams & Dunlop 1993, eqs. 27 and 32) is the
// 27-point weighted combination of the indefinite integrals, evaluated in
// double precision exactly as physics/newell.cu:7-139 does, and summed over the
// PBC images (2r+1 per periodic axis) as physics/strayfieldkernel.cu:25-56 does
// -- here the image sum is also FP64.  The integrals of the 27 points are shared:
// they are evaluated once per lattice point (k_newell_lattice; neighbouring
// displacements and periodic images meet the same points) and combined per
// displacement in the order of the direct sum (k_newell_from_lattice).  It is
// evaluated once per octant point |r| (the tensor is even in every axis for
// xx/yy/zz and odd in the axes its off-diagonal indices name).  The spectrum of
// such a tensor is real, and each axis is a cosine or sine transform of the
// octant values alone: three passes (k_kernel_axis) of FP64 transforms in shared
// memory take the octant table to the symmetry-reduced spectrum
// (kx in [0,Px/2], ky in [0,Py/2], kz in [0,Pz/2]), stored in FP32 with the
// convolution prefactor -mu0/(Px Py Pz) folded in.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace mpx {

__device__ __forceinline__ double nxx_indef(int ix, int iy, int iz, double cx, double cy, double cz) {
  const double x = ix * cx, y = iy * cy, z = iz * cz;
  const double R = sqrt(x * x + y * y + z * z);
  double r = 0;
  if (ix != 0 || iz != 0) r += (y / 2) * (z * z - x * x) * asinh(y / sqrt(x * x + z * z));
  if (ix != 0 || iy != 0) r += (z / 2) * (y * y - x * x) * asinh(z / sqrt(x * x + y * y));
  if (ix != 0) r -= x * y * z * atan((y * z) / (x * R));
  r += (1. / 6.) * (2 * x * x - y * y - z * z) * R;
  return r;
}

__device__ __forceinline__ double nxy_indef(int ix, int iy, int iz, double cx, double cy, double cz) {
  if (iy == 0 || ix == 0) return 0.0;
  const double x = ix * cx, y = iy * cy, z = iz * cz;
  const double R = sqrt(x * x + y * y + z * z);
  double r = 0;
  r += (x * y * z) * asinh(z / sqrt(x * x + y * y));
  r += (y / 6) * (3 * z * z - y * y) * asinh(x / sqrt(y * y + z * z));
  r += (x / 6) * (3 * z * z - x * x) * asinh(y / sqrt(x * x + z * z));
  r -= (z * y * y / 2) * atan((x * z) / (y * R));
  r -= (z * x * x / 2) * atan((y * z) / (x * R));
  r -= x * y * R / 3;
  if (iz != 0) r -= (z * z * z / 6) * atan((x * y) / (z * R));
  return r;
}

__device__ __forceinline__ int newell_w(int dx, int dy, int dz) {
  const int s = dx * dx + dy * dy + dz * dz;
  return s == 0 ? 8 : s == 1 ? -4 : s == 2 ? 2 : -1;
}

static __device__ double newell_nxx(int ix, int iy, int iz, double cx, double cy, double cz) {
  double r = 0;
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dz = -1; dz <= 1; ++dz)
        r += newell_w(dx, dy, dz) * nxx_indef(ix + dx, iy + dy, iz + dz, cx, cy, cz);
  return r / (4 * M_PI * cx * cy * cz);
}

static __device__ double newell_nxy(int ix, int iy, int iz, double cx, double cy, double cz) {
  if (ix == 0 || iy == 0) return 0;
  double r = 0;
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dz = -1; dz <= 1; ++dz)
        r += newell_w(dx, dy, dz) * nxy_indef(ix + dx, iy + dy, iz + dz, cx, cy, cz);
  return r / (4 * M_PI * cx * cy * cz);
}

// component c (xx, yy, zz, xy, xz, yz) at displacement (x, y, z) cells
static __device__ double newell_comp(int c, int x, int y, int z, double cx, double cy, double cz) {
  switch (c) {
    case 0: return newell_nxx(x, y, z, cx, cy, cz);
    case 1: return newell_nxx(y, z, x, cy, cz, cx);
    case 2: return newell_nxx(z, x, y, cz, cx, cy);
    case 3: return newell_nxy(x, y, z, cx, cy, cz);
    case 4: return newell_nxy(x, z, y, cx, cz, cy);
    default: return newell_nxy(y, z, x, cy, cz, cx);
  }
}

struct KernelGeom {
  int n[3];      // source/destination grid size
  int mg[3];     // mastergrid size (image period)
  int pbc[3];    // image repetitions
  double cs[3];  // cell size
};

// Table of N_c at the displacements O + j, j < K per axis (layout [c][z][y][x]),
// each with its images, evaluated point by point: where the lattice (below) of even
// one image does not fit its share of the memory.
template <typename T>
__global__ void k_newell_direct(T* __restrict__ out, KernelGeom g, int K0, int K1, int K2, int O0, int O1, int O2,
                                int ncomp) {
  const long long total = (long long)K0 * K1 * K2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int x0 = O0 + (int)(t % K0);
    const int y0 = O1 + (int)((t / K0) % K1);
    const int z0 = O2 + (int)(t / ((long long)K0 * K1));
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int i = -g.pbc[0]; i <= g.pbc[0]; ++i)
      for (int j = -g.pbc[1]; j <= g.pbc[1]; ++j)
        for (int k = -g.pbc[2]; k <= g.pbc[2]; ++k)
#pragma unroll 1
          for (int c = 0; c < ncomp; ++c)
            v[c] += newell_comp(c, x0 + i * g.mg[0], y0 + j * g.mg[1], z0 + k * g.mg[2], g.cs[0], g.cs[1], g.cs[2]);
    for (int c = 0; c < ncomp; ++c) out[c * total + t] = (T)v[c];
  }
}

// The lattice points |q| = a0 + p, p < len per axis (q in cells), that a table of
// displacements meets: every displacement, its images included, and their neighbours.
struct NewellLattice {
  int a0[3], len[3];
};
// Periodic images lo .. hi per axis.
struct NewellImages {
  int lo[3], hi[3];
};

// Axes (u, v, w) of the arguments of component c (newell_comp's permutations).
__device__ __forceinline__ void newell_axes(int c, int& u, int& v, int& w) {
  u = c == 0 || c == 3 || c == 4 ? 0 : c == 2 ? 2 : 1;
  v = c == 0 || c == 3 ? 1 : c == 2 ? 0 : 2;
  w = 3 - u - v;
}

// Indefinite integrals of components c0 .. c0 + nc - 1 at every lattice point
// (layout [c - c0][z][y][x]).  FP64 arithmetic bounds it (3 to 5 transcendental
// functions per value); sharing the values takes 27 evaluations per displacement
// and component to about one.
static __global__ void k_newell_lattice(double* __restrict__ lat, KernelGeom g, NewellLattice L, int c0, int nc) {
  const long long total = (long long)L.len[0] * L.len[1] * L.len[2];
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total * nc;
       t += (long long)gridDim.x * blockDim.x) {
    const int c = c0 + (int)(t / total);
    const long long e = t % total;
    const int q[3] = {L.a0[0] + (int)(e % L.len[0]), L.a0[1] + (int)((e / L.len[0]) % L.len[1]),
                      L.a0[2] + (int)(e / ((long long)L.len[0] * L.len[1]))};
    int u, v, w;
    newell_axes(c, u, v, w);
    const int qu = u == 0 ? q[0] : u == 1 ? q[1] : q[2], qv = v == 0 ? q[0] : v == 1 ? q[1] : q[2];
    const int qw = w == 0 ? q[0] : w == 1 ? q[1] : q[2];
    lat[t] = c < 3 ? nxx_indef(qu, qv, qw, g.cs[u], g.cs[v], g.cs[w]) : nxy_indef(qu, qv, qw, g.cs[u], g.cs[v], g.cs[w]);
  }
}

// k_newell_direct's table of components c0 .. c0 + nc - 1 from the lattice.  The
// integrals of the diagonal components are even in every argument, those of the
// off-diagonal ones odd in the first two; the 27 terms and the images are added
// in the order of the direct sum.  The images may come in several parts of that
// order: `acc` (components from ca on) holds the sum of the parts before this one
// unless it is the first, and takes it unless this one is the last.
template <typename T>
__global__ void k_newell_from_lattice(T* out, double* acc, int ca, bool first, bool last,
                                      const double* __restrict__ lat, KernelGeom g, NewellLattice L, NewellImages I,
                                      int c0, int nc, int K0, int K1, int K2, int O0, int O1,
                                      int O2) {
  const long long total = (long long)K0 * K1 * K2, ltot = (long long)L.len[0] * L.len[1] * L.len[2];
  const long long ls[3] = {1, L.len[0], (long long)L.len[0] * L.len[1]};
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total * nc;
       t += (long long)gridDim.x * blockDim.x) {
    const int c = c0 + (int)(t / total);
    const long long e = t % total;
    const int d[3] = {O0 + (int)(e % K0), O1 + (int)((e / K0) % K1), O2 + (int)(e / ((long long)K0 * K1))};
    int u, v, w;
    newell_axes(c, u, v, w);
    const double norm = 4 * M_PI * g.cs[u] * g.cs[v] * g.cs[w];
    const double* __restrict__ F = lat + (c - c0) * ltot;
    double sum = first ? 0 : acc[(c - ca) * total + e];
    for (int i = I.lo[0]; i <= I.hi[0]; ++i)
      for (int j = I.lo[1]; j <= I.hi[1]; ++j)
        for (int k = I.lo[2]; k <= I.hi[2]; ++k) {
          const int q[3] = {d[0] + i * g.mg[0], d[1] + j * g.mg[1], d[2] + k * g.mg[2]};
          const int qu = u == 0 ? q[0] : u == 1 ? q[1] : q[2], qv = v == 0 ? q[0] : v == 1 ? q[1] : q[2];
          const int qw = w == 0 ? q[0] : w == 1 ? q[1] : q[2];
          double r = 0;
          if (c < 3 || (qu != 0 && qv != 0)) {
            const long long su = ls[u], sv = ls[v], sw = ls[w];
#pragma unroll
            for (int du = -1; du <= 1; ++du)
#pragma unroll
              for (int dv = -1; dv <= 1; ++dv)
#pragma unroll
                for (int dw = -1; dw <= 1; ++dw) {
                  double f = F[su * (abs(qu + du) - L.a0[u]) + sv * (abs(qv + dv) - L.a0[v]) +
                               sw * (abs(qw + dw) - L.a0[w])];
                  if (c >= 3 && ((qu + du < 0) != (qv + dv < 0))) f = -f;
                  r += newell_w(du, dv, dw) * f;
                }
            r /= norm;
          }
          sum += r;
        }
    if (last) out[c * total + e] = (T)sum;
    else acc[(c - ca) * total + e] = sum;
  }
}

// The same table from one over absolute displacements: entry j of the output
// is displacement O + j (K per axis); the input holds |d| = A + a (a < L per
// axis), same layout.  Diagonal components are even in every displacement
// component, xy odd in x and y, xz in x and z, yz in y and z, also after the sum
// over periodic images (their repetitions run over -p .. p), so each output is
// an input entry times the signs of its odd components.
static __global__ void k_newell_expand_abs(float* __restrict__ out, const float* __restrict__ abs_tab, int K0, int K1,
                                    int K2, int O0, int O1, int O2, int A0, int A1, int A2, int L0, int L1, int L2) {
  const long long total = (long long)K0 * K1 * K2, ltot = (long long)L0 * L1 * L2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = O0 + (int)(t % K0);
    const int y = O1 + (int)((t / K0) % K1);
    const int z = O2 + (int)(t / ((long long)K0 * K1));
    const long long p = ((long long)(abs(z) - A2) * L1 + (abs(y) - A1)) * L0 + (abs(x) - A0);
    const float sx = x < 0 ? -1.f : 1.f, sy = y < 0 ? -1.f : 1.f, sz = z < 0 ? -1.f : 1.f;
    out[t] = abs_tab[p];
    out[total + t] = abs_tab[ltot + p];
    out[2 * total + t] = abs_tab[2 * ltot + p];
    out[3 * total + t] = (sx * sy) * abs_tab[3 * ltot + p];
    out[4 * total + t] = (sx * sz) * abs_tab[4 * ltot + p];
    out[5 * total + t] = (sy * sz) * abs_tab[5 * ltot + p];
  }
}

// One axis of the kernel transform.  A line of n octant values f_j (j = 0 .. n-1)
// stands for the circular sequence of length P with x[j] = f_j, x[P - j] = +-f_j
// (even or odd component); its transform is real, f_0 + 2 sum f_j cos(2 pi j k/P),
// or -i times the real 2 sum f_j sin(2 pi j k/P).  Two lines share one complex
// FFT.  `inner` lines lie si apart, (o1, o2) groups of them further; elements of a
// line lie sj apart.  Output k in [0, P/2] likewise.
struct KernelAxis {
  int n, P, inner, n2;                 // n2: number of o2 groups
  long long sj, si, so1, so2;          // input strides
  long long tk, ti, to1, to2;          // output strides
  unsigned odd;                        // bit c: component c (o1) is odd along this axis
  double scale[6];                     // factor per component
};

// Stockham pass of radix R over `nl` complex lines of length P (line l at l*P),
// from a to b; tw[m] = exp(-2 pi i m / P).
template <int R>
__device__ __forceinline__ void fft64_pass(const double2* a, double2* b, int nl, int P, int Ns, const double2* tw) {
  const int NB = P / R, total = nl * NB, step = P / (Ns * R);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int l = t / NB, j = t - l * NB, k = j % Ns;
    double2 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double2 v = a[l * P + j + r * NB], w = tw[r * k * step];
      x[r] = r == 0 ? v : make_double2(v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x);
    }
    double2* o = b + l * P + (j - k) * R + k;
    if constexpr (R == 2) {
      o[0] = make_double2(x[0].x + x[1].x, x[0].y + x[1].y);
      o[Ns] = make_double2(x[0].x - x[1].x, x[0].y - x[1].y);
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        double2 y = x[0];
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const double2 w = tw[((q * r) % R) * NB];
          y.x += x[r].x * w.x - x[r].y * w.y;
          y.y += x[r].x * w.y + x[r].y * w.x;
        }
        o[q * Ns] = y;
      }
    }
  }
  __syncthreads();
}

// Blocks of TL complex lines (2 TL real ones); dynamic shared memory
// (2 TL + 1) P double2.  Grid: o1 * n2 * ceil(inner / (2 TL)).  Bound by shared
// memory (log2 P passes over 16-byte values); the transforms touch the octant's
// lines only, about an eighth of the padded grid, in 3 launches for all components.
template <typename TO>
__global__ void __launch_bounds__(256) k_kernel_axis(const double* __restrict__ in, TO* __restrict__ out, KernelAxis A,
                                                     int TL) {
  extern __shared__ double2 sd[];
  const int P = A.P, nt = (A.inner + 2 * TL - 1) / (2 * TL);
  const int tile = blockIdx.x % nt, o2 = (blockIdx.x / nt) % A.n2, o1 = blockIdx.x / (nt * A.n2);
  const int i0 = tile * 2 * TL, ni = min(2 * TL, A.inner - i0);
  const bool odd = (A.odd >> o1) & 1;
  double2 *a = sd, *b = sd + TL * P, *tw = sd + 2 * TL * P;
  double* ar = reinterpret_cast<double*>(a);
  for (int t = threadIdx.x; t < P; t += blockDim.x) {
    double s, c;
    sincospi(-2.0 * t / P, &s, &c);
    tw[t] = make_double2(c, s);
  }
  for (int t = threadIdx.x; t < TL * P; t += blockDim.x) a[t] = make_double2(0, 0);
  __syncthreads();
  const double* src = in + o1 * A.so1 + o2 * A.so2 + i0 * A.si;
  for (int t = threadIdx.x; t < ni * A.n; t += blockDim.x) {  // consecutive threads along the unit stride
    const int i = A.sj == 1 ? t / A.n : t % ni, j = A.sj == 1 ? t % A.n : t / ni;
    const double v = src[j * A.sj + i * A.si];
    double* line = ar + 2 * (i >> 1) * P + (i & 1);  // real part: even lines, imaginary: odd lines
    if (j == 0) {
      line[0] = odd ? 0.0 : v;
    } else {
      line[2 * j] = v;
      line[2 * (P - j)] = odd ? -v : v;
    }
  }
  __syncthreads();
  int Ns = 1, rest = P;
  while (rest % 3 == 0) {
    fft64_pass<3>(a, b, TL, P, Ns, tw);
    double2* x = a;
    a = b;
    b = x;
    Ns *= 3;
    rest /= 3;
  }
  while (rest > 1) {
    fft64_pass<2>(a, b, TL, P, Ns, tw);
    double2* x = a;
    a = b;
    b = x;
    Ns *= 2;
    rest /= 2;
  }
  const int H = P / 2 + 1;
  TO* dst = out + o1 * A.to1 + o2 * A.to2 + i0 * A.ti;
  const double sc = A.scale[o1];
  for (int t = threadIdx.x; t < ni * H; t += blockDim.x) {
    const int i = A.tk == 1 ? t / H : t % ni, k = A.tk == 1 ? t % H : t / ni;
    const double2 X = a[(i >> 1) * P + k];
    // even: X = A + i B; odd: X = -i A + B of the two real transforms A, B
    const double v = odd ? ((i & 1) ? X.x : -X.y) : ((i & 1) ? X.y : X.x);
    dst[k * A.tk + i * A.ti] = (TO)(sc * v);
  }
}

}  // namespace mpx
