// stages.cuh -- the Runge-Kutta kernels beside the demag passes: local terms
// without demag, the stage combination, and the step controller.  Included by
// xpass.cu only (with the x passes they read the Butcher tableau of that file).
#pragma once
#include "kernels.cuh"

namespace mpx {

// Local terms only (no demag): same tiles, no dynamic shared memory.
static __global__ void __launch_bounds__(256) k_local(const MagnetDev* __restrict__ mags, GroupDev* __restrict__ groups,
                                               const Work* __restrict__ work, EpiArgs ea) {
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, ea.gate, ea.stage)) return;
  const int nx = M.n[0], ny = M.n[1];
  const float* m = ea.msrc ? ea.msrc : stage_m(M, G, ea.stage);
  double en = 0.0, tn = 0.0;
  const int rowbase = nx * (wk.y0 + ny * wk.z);
  const float rn = 1.0f / (float)nx;
  for (int e = threadIdx.x; e < wk.ty * nx; e += blockDim.x) {
    const int yl = tile_row(e, nx, rn), x = e - yl * nx;
    double a = 0.0, b = 0.0;
    epilogue_cell(M, G, ea, m, x, wk.y0 + yl, wk.z, rowbase + e, f3(0, 0, 0), a, b);
    en = (a > en || a != a) ? a : en;
    tn = fmax(tn, b);
  }
  if (ea.fsal_err) block_max2(en, tn, &groups[M.group].err_bits, &groups[M.group].tmax_bits);
}

// Stage combination without a demag pass (writes the stage state xs), or the
// final combination of a non-FSAL method with its error estimate
// (core/rungekutta.cpp:123-151).
static __global__ void __launch_bounds__(256) k_combine(const MagnetDev* __restrict__ mags, GroupDev* __restrict__ groups,
                                                 const Work* __restrict__ work, int stage, int final_b1) {
  __shared__ MagnetDev M;
  __shared__ GroupDev G;
  const Work wk = work[blockIdx.x];
  if (!load_descs(M, G, mags, groups, wk.mag, 1, 1)) return;
  const int nx = M.n[0], ny = M.n[1], N = M.N;
  float* xs = M.buf[G.map[1]];
  const float* x0 = M.buf[G.map[0]];
  double en = 0.0;
  const int rowbase = nx * (wk.y0 + ny * wk.z);
  for (int e = threadIdx.x; e < wk.ty * nx; e += blockDim.x) {
    const int i = rowbase + e;
    if (!in_geom(M, i)) {
      store3(xs, N, i, load3(x0, N, i));
      continue;
    }
    store3(xs, N, i, combine_cell(M, G, stage, i, final_b1 != 0));
    if (final_b1 && G.adaptive) {
      float3 ev = f3(0, 0, 0);
      for (int j = 0; j < c_tab.S; ++j) {
        const float cf = (float)(G.dt * (c_tab.b1[j] - c_tab.b2[j]));
        const float3 kj = load3(M.buf[G.map[2 + j]], N, i);
        ev = f3(ev.x + cf * kj.x, ev.y + cf * kj.y, ev.z + cf * kj.z);
      }
      const double a = sqrt((double)ev.x * ev.x + (double)ev.y * ev.y + (double)ev.z * ev.z);
      en = (a > en || a != a) ? a : en;
    }
  }
  if (final_b1) block_max2(en, 0.0, &groups[M.group].err_bits, &groups[M.group].tmax_bits);
}

// --------------------------------------------------------------- controller
// core/rungekutta.cpp:60-82 and core/timesolver.cpp:60-111, one thread per group,
// in FP64.  Also runs the run()/steps() state machine on the device.
// Sampled run: time point samp_k has been reached.  Its row (and the rows of
// the next points that need no step, as run(t_k - t) with t_k <= t takes none)
// become due with the time; the next point that needs steps is armed as run()
// arms its end (core/timesolver.cpp:100-109).  Returns false when no point is
// left.
__device__ __forceinline__ bool sample_advance(GroupDev& G) {
  G.samp_lo = G.samp_k;
  do {
    G.samp_out[(size_t)G.samp_k * G.samp_row] = G.t;
    ++G.samp_k;
  } while (G.samp_k < G.samp_n && !(G.samp_t[G.samp_k] - G.t > 0.0));
  G.samp_hi = G.samp_k;
  if (G.samp_k >= G.samp_n) return false;
  G.phase = 0;
  G.t_stop = G.t + (G.samp_t[G.samp_k] - G.t);
  if (!(G.t < G.t_stop - G.dt)) {
    G.phase = 1;
    G.dt_saved = G.dt;
    G.dt = G.t_stop - G.t;
  }
  return true;
}

static __global__ void k_controller(GroupDev* __restrict__ groups, int ngroups) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ngroups) return;
  GroupDev& G = groups[g];
  if (G.status != GS_RUNNING) return;
  G.samp_lo = G.samp_hi;  // the rows of the previous attempt have been written
  const double err = __longlong_as_double((long long)G.err_bits);
  const double tmax = __longlong_as_double((long long)G.tmax_bits);
  G.err_bits = 0ull;
  G.tmax_bits = 0ull;
  G.attempts++;
  const double dt = G.dt;
  bool success = true;
  if (G.adaptive) {
    success = err < G.max_error;
    double corr = success ? pow(G.max_error / err, 1.0 / (c_tab.order2 + 1))
                          : pow(G.max_error / err, 1.0 / (c_tab.order1 + 1));
    if (isnan(corr)) corr = 1.0;
    corr *= G.headroom;
    corr = corr > G.upper ? G.upper : corr;
    corr = corr < G.lower ? G.lower : corr;
    G.dt = dt * corr;
    if (isnan(err)) {  // the reference would retry forever; fail the solve instead
      G.status = GS_FAILED;
      G.finished_flag = 1;
      return;
    }
  }
  if (!success) {
    G.rejected++;
    G.k0_valid = G.thermal ? 0 : 1;  // with noise k0 depends on dt (noise / sqrt(dt))
    return;
  }
  // accept: t = t0 + dt; x0 <- x_new; FSAL: k0 <- k_{S-1}
  G.t += dt;
  G.steps++;
  const int t0 = G.map[0];
  G.map[0] = G.map[1];
  G.map[1] = t0;
  if (c_tab.fsal) {
    const int k0 = G.map[2];
    G.map[2] = G.map[2 + c_tab.S - 1];
    G.map[2 + c_tab.S - 1] = k0;
    G.k0_valid = G.thermal ? 0 : 1;  // a new step draws new noise
  } else {
    G.k0_valid = 0;
  }
  bool done = false;
  if (G.phase == 1) {
    done = true;
    if (!G.adaptive) G.dt = G.dt_saved;
    if (G.mode == 2) done = !sample_advance(G);
  } else if (G.mode == 1) {
    if (--G.steps_left <= 0) done = true;
  } else {
    if (G.torque_stop > 0.0 && c_tab.fsal && tmax / (double)GAMMA_LL < G.torque_stop) {
      done = true;
    } else if (!(G.t < G.t_stop - G.dt)) {
      G.phase = 1;
      G.dt_saved = G.dt;
      G.dt = G.t_stop - G.t;
    }
  }
  if (done) {
    G.status = GS_FINISHED;
    G.finished_flag = 1;
    G.phase = 0;
  }
}

}  // namespace mpx
