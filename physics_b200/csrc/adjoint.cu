// Reverse-mode adjoint of the f64 plain SPH step
// (FluidWorld<f64>::step, crates/phy-fluid/src/sph/world.rs:183-397).
//
// The forward step of one particle i (d = x_j - x_i, r = |d|, u = d / r,
// dv = v_j - v_i, j over the step's neighbours with 0 < r < h):
//   rho_i   = sum_{r<h} m_j W(r)                       (self included)
//   p_i     = k max(0, rho_i - rho0),  pi_i = p_i / rho_i^2
//   fp_i    = sum u m_i m_j (pi_i + pi_j) G(r)          G = spiky gradient
//   fv_i    = sum dv m_i m_j / rho_j L(r)               L = viscosity Laplacian
//   xs_i    = sum dv m_j / rho_j W(r)
//   s_i     = sum |dv| / (r + 1e-4) m_j / rho_j
//   mu_i    = visc_k[m] max(s_i, shear_min)^(n-1)
//   acc_i   = (fp_i + fv_i mu_i) / rho_i
//   v'      = v + ((acc + g) + b) dt + xs eps;  x' = x + v' dt;  walls clamp
//             x' and reflect v' with damping.
// The reverse sweep holds the step's neighbour sets and every branch (wall
// contacts, max(0, .), shear_min) fixed, as the forward took them, and is
// exact for that piecewise-smooth map.
//
// Gradient flow (one reverse step, all arrays in the step's sorted order):
//   k_adj_integrate   dL/dx', dL/dv' -> direct dL/dx, dL/dv, the seeds of the
//                     pair sums (dL/dfp, dL/dfv, dL/dxs, dL/ds), the direct
//                     dL/drho and the visc_k[0] term;
//   k_adj_force       for each particle i, over its neighbours j, the
//                     derivatives of i's own pair terms (i's seeds) and of j's
//                     pair terms that involve i (j's seeds) — the neighbour
//                     relation is symmetric, so every contribution to i is
//                     gathered by i and no atomics are needed; its epilogue
//                     closes dL/drho_i through pi_i and p_i and the stiffness
//                     term;
//   k_adj_density     the density sums: dL/dx_i += sum W'(r) (x_i - x_j) / r
//                     (m_j dL/drho_i + m_i dL/drho_j), then the scatter back to
//                     insertion order.
// The parameter gradients are per-particle terms summed by a fixed-order
// reduction, so a gradient repeats bit-exactly run to run.
//
// The forward quantities the reverse needs (sorted state, rho, p, pi, m/rho,
// acc, xsph, mu, fv and s, the cell ranges) are recorded as the forward
// steps run, or by re-running them from checkpoints; the wall decisions are
// recomputed here with the forward's exact operation order.
#include <cuda_runtime.h>

#include "adjoint.h"

namespace phy {

namespace {

constexpr int kThreads = 128;
constexpr double kShearEps = 1e-4;  // world.rs:259 (r + 1e-4 in the strain proxy)

__device__ __forceinline__ double norm2(double x, double y, double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Kernel values and radial derivatives at r (< h0; zero beyond, as the
// forward's kernels).
struct KernelDerivs {
  double G, Gp, L, Lp, W, Wp;
};

__device__ __forceinline__ KernelDerivs kernel_derivs(const StepConsts& c, double r) {
  KernelDerivs k;
  if (r >= c.h0) {
    k.G = k.Gp = k.L = k.Lp = k.W = k.Wp = 0.0;
    return k;
  }
  const double hr = c.h0 - r;
  const double q = c.h0sq - r * r;
  k.G = c.spiky_c * hr * hr;
  k.Gp = -2.0 * c.spiky_c * hr;
  k.L = c.lap_c * hr;
  k.Lp = -c.lap_c;
  k.W = c.poly6_c * q * q * q;
  k.Wp = -6.0 * c.poly6_c * r * q * q;
  return k;
}

// The pair kernels' operands of a slot as 32-byte parts, one array each: x and
// mass; v and m/rho; the seeds P and p/rho^2; Q and sig; Y.  A neighbour is
// five loads instead of seventeen.
struct d4 {
  double x, y, z, w;
};
__device__ __forceinline__ d4 load_part(const AdjWork& w, int part, size_t n, int j) {
  const double* p = w.rec + 4 * (part * n + (size_t)j);
  d4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void store_part(const AdjWork& w, int part, size_t n, int j, double x, double y, double z,
                                           double v) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(w.rec + 4 * (part * n + (size_t)j)), "d"(x), "d"(y),
               "d"(z), "d"(v)
               : "memory");
}

__global__ void __launch_bounds__(kThreads) k_adj_integrate(StepConsts c, AdjTape t, AdjWork w) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.n) return;
  const uint32_t ins = t.id[s];
  const double x3[3] = {t.x[0][s], t.x[1][s], t.x[2][s]};
  const double v3[3] = {t.v[0][s], t.v[1][s], t.v[2][s]};
  const double acc3[3] = {t.acc[0][s], t.acc[1][s], t.acc[2][s]};
  const double xs3[3] = {t.xsph[0][s], t.xsph[1][s], t.xsph[2][s]};
  double accb[3], P[3], Q[3], Y[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // The forward's integrate and enforce_bounds, operation for operation, to
    // recover the wall decision (body accelerations are zero on a tape).
    const double ak = __dadd_rn(__dadd_rn(acc3[a], c.g[a]), 0.0);
    double v = __dadd_rn(v3[a], __dmul_rn(ak, c.dt));
    v = __dadd_rn(v, __dmul_rn(xs3[a], c.xsph_eps));
    const double x = __dadd_rn(x3[a], __dmul_rn(v, c.dt));
    const bool wall = x < c.lo[a] || x > c.hi[a];
    const double xb_out = w.gx_ins[a][ins], vb_out = w.gv_ins[a][ins];
    const double xb1 = wall ? 0.0 : xb_out;
    double vb2 = wall ? -c.damp * vb_out : vb_out;
    vb2 += xb1 * c.dt;
    w.gx[a][s] = xb1;
    w.gv[a][s] = vb2;
    Y[a] = vb2 * c.xsph_eps;
    accb[a] = vb2 * c.dt;
  }
  const double rho = t.rho[s], mu = t.mu[s];
  double rbar = 0.0, mub = 0.0;
  if (rho > 0.0) {
    const double inv = 1.0 / rho;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      P[a] = accb[a] * inv;
      Q[a] = accb[a] * mu * inv;
      mub += accb[a] * t.fv[a][s] * inv;
      rbar -= accb[a] * acc3[a] * inv;
    }
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      P[a] = 0.0;
      Q[a] = 0.0;
    }
  }
  // mu = kc * (n == 1 ? 1 : max(s, shear_min)^(n-1))  (world.rs:319-327)
  const uint32_t m = t.mat[s];
  const int midx = (int)m < c.n_visc_k ? (int)m : 0;
  double kc, nn;
  material_coeffs(c, midx, kc, nn);
  const double ex = nn - 1.0;
  const double shear = t.shear[s];
  const double sreg = shear > c.shear_min ? shear : c.shear_min;
  const double fac = ex == 0.0 ? 1.0 : pow(sreg, ex);
  w.cc[s] = midx == 0 ? mub * fac : 0.0;
  const double sig = (ex != 0.0 && shear > c.shear_min) ? mub * kc * ex * pow(sreg, ex - 1.0) : 0.0;
  const size_t n = (size_t)c.n;
  store_part(w, 0, n, s, x3[0], x3[1], x3[2], t.mass[s]);
  store_part(w, 1, n, s, v3[0], v3[1], v3[2], t.mr[s]);
  store_part(w, 2, n, s, P[0], P[1], P[2], t.pr2[s]);
  store_part(w, 3, n, s, Q[0], Q[1], Q[2], sig);
  store_part(w, 4, n, s, Y[0], Y[1], Y[2], 0.0);
  w.rbar[s] = rbar;
}

// Lanes per particle of the pair kernels: a particle's neighbours are dealt
// round-robin to kLanes consecutive lanes of a warp, whose partial sums are
// then combined by a fixed shuffle tree (deterministic).  Two lanes, since
// more of them drift apart in their list rows (65,536 particles, force and
// density pass: 75 + 26 us with one lane, 66 + 18 with two, 71 + 24 with four,
// 91 + 30 with eight); four in small worlds, where the longest lane is what
// takes the time (a whole reverse step with four and two lanes: 512 particles
// 31 / 43 us, 3,920 36 / 42, 15,488 41 / 49, 26,656 50 / 56, 32,768 57 / 57,
// 65,600 110 / 97, 196,608 252 / 230).
constexpr int kLanesBelow = 30000;

// Visits lane `q`'s share of the step's force/density neighbours of slot i:
// its recorded list, or the 27 cells when the list overflowed (and, for a
// particle outside the grid box, nothing).  `f(j)` applies the pair tests.
template <int kLanes, class F>
__device__ __forceinline__ void for_each_listed(const StepConsts& c, const AdjTape& t, int i, int q, double xi,
                                                double yi, double zi, F&& f) {
  const uint32_t cnt = t.nbr_count[i];
  if (cnt <= (uint32_t)kMaxNeighbors) {
    // The next index is loaded while this neighbour is computed.
    uint32_t j = (uint32_t)q < cnt ? t.nbr[(size_t)q * c.n + i] : 0u;
    for (uint32_t k = q; k < cnt; k += kLanes) {
      const int jc = (int)j;
      if (k + kLanes < cnt) j = t.nbr[(size_t)(k + kLanes) * c.n + i];
      f(jc);
    }
    return;
  }
  const long long kx = key_axis(xi, c.inv_cell), ky = key_axis(yi, c.inv_cell), kz = key_axis(zi, c.inv_cell);
  if (!cell_interior(c, kx, ky, kz)) return;
  const int base = cell_linear(c, kx - 1, ky - 1, kz - 1);
  for (int di = 0; di < 3; ++di)
    for (int dj = 0; dj < 3; ++dj) {
      const int c0 = base + (di * c.ncy + dj) * c.ncz;
      const int s0 = (int)t.cell_start[c0], e0 = (int)t.cell_start[c0 + 3];
      for (int j = s0 + q; j < e0; j += kLanes)
        if (j != i) f(j);
    }
}

// Sum over the kLanes lanes of a particle (all lanes receive the total).
template <int kLanes>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 128 registers (four blocks per SM) spill nothing and beat the 146 that the
// compiler would take: 66 -> 64 us; 102 of them spill (101 us).
template <int kLanes>
__global__ void __launch_bounds__(kThreads, 4) k_adj_force(StepConsts c, AdjTape t, AdjWork w) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = g / kLanes, q = g % kLanes;
  const bool live = i < c.n;  // whole particles per warp: kLanes divides 32
  const int ii = live ? i : 0;
  const size_t n = (size_t)c.n;
  const d4 xo = load_part(w, 0, n, ii), vo = load_part(w, 1, n, ii), po = load_part(w, 2, n, ii),
           qo = load_part(w, 3, n, ii), yo = load_part(w, 4, n, ii);
  const double xi = xo.x, yi = xo.y, zi = xo.z, vxi = vo.x, vyi = vo.y, vzi = vo.z;
  const double m_i = xo.w, pr2_i = po.w, mr_i = vo.w;
  const double Pi[3] = {po.x, po.y, po.z}, Qi[3] = {qo.x, qo.y, qo.z}, Yi[3] = {yo.x, yo.y, yo.z};
  const double sig_i = qo.w;
  double gx[3] = {0.0, 0.0, 0.0}, gv[3] = {0.0, 0.0, 0.0};
  double pibar = 0.0, rsum = 0.0;
  if (live) for_each_listed<kLanes>(c, t, i, q, xi, yi, zi, [&](int j) {
    // The forward's neighbour test (d = p_j - p_i, world.rs:295-299).
    const d4 xj = load_part(w, 0, n, j), vj = load_part(w, 1, n, j), pj = load_part(w, 2, n, j),
             qj = load_part(w, 3, n, j), yj = load_part(w, 4, n, j);
    const double d[3] = {__dsub_rn(xj.x, xi), __dsub_rn(xj.y, yi), __dsub_rn(xj.z, zi)};
    const double r2 = norm2(d[0], d[1], d[2]);
    if (r2 > c.r2_guard) return;
    const double r = __dsqrt_rn(r2);
    if (r >= c.h || r <= 0.0) return;
    const KernelDerivs k = kernel_derivs(c, r);
    const double inv_r = __drcp_rn(r);
    const double u[3] = {d[0] * inv_r, d[1] * inv_r, d[2] * inv_r};
    const double dv[3] = {vj.x - vxi, vj.y - vyi, vj.z - vzi};
    const double dv2 = dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2];
    const double inv_dvn = dv2 > 0.0 ? rsqrt(dv2) : 0.0;
    const double dvn = dv2 * inv_dvn;
    const double m_j = xj.w, mr_j = vj.w;
    const double mm = m_i * m_j;
    const double A = mm * (pr2_i + pj.w);
    const double inv_re = __drcp_rn(r + kShearEps);
    const double Pj[3] = {pj.x, pj.y, pj.z}, Qj[3] = {qj.x, qj.y, qj.z}, Yj[3] = {yj.x, yj.y, yj.z};
    const double sig_j = qj.w;
    // Own terms (i's seeds): variables d, dv, pi_i, pi_j, rho_j.
    const double uP = u[0] * Pi[0] + u[1] * Pi[1] + u[2] * Pi[2];
    const double dvQ = dv[0] * Qi[0] + dv[1] * Qi[1] + dv[2] * Qi[2];
    const double dvY = dv[0] * Yi[0] + dv[1] * Yi[1] + dv[2] * Yi[2];
    const double B = m_i * mr_j;  // m_i m_j / rho_j
    const double AGr = A * k.G * inv_r;
    const double radial_own = (A * k.Gp - AGr) * uP + dvQ * B * k.Lp + dvY * mr_j * k.Wp -
                              sig_i * dvn * mr_j * inv_re * inv_re;
    const double sv_own = sig_i * mr_j * inv_re * inv_dvn;
    // Cross terms (j's seeds; from j's side d' = -d, u' = -u, dv' = -dv, and
    // rho_i is the neighbour density).
    const double uPj = -(u[0] * Pj[0] + u[1] * Pj[1] + u[2] * Pj[2]);
    const double dvQj = -(dv[0] * Qj[0] + dv[1] * Qj[1] + dv[2] * Qj[2]);
    const double dvYj = -(dv[0] * Yj[0] + dv[1] * Yj[1] + dv[2] * Yj[2]);
    const double Bi = m_j * mr_i;  // m_i m_j / rho_i
    const double radial_x = (A * k.Gp - AGr) * uPj + dvQj * Bi * k.Lp + dvYj * mr_i * k.Wp -
                            sig_j * dvn * mr_i * inv_re * inv_re;
    const double sv_x = sig_j * mr_i * inv_re * inv_dvn;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // d(own)/d d and d(own)/d dv; x_i enters d with a minus sign.
      const double gd_own = radial_own * u[a] + AGr * Pi[a];
      const double gdv_own = Qi[a] * B * k.L + Yi[a] * mr_j * k.W + sv_own * dv[a];
      // d(cross)/d d' (u' = -u) and d(cross)/d dv' (dv' = -dv); x_i enters d' with a plus sign.
      const double gd_x = -radial_x * u[a] + AGr * Pj[a];
      const double gdv_x = Qj[a] * Bi * k.L + Yj[a] * mr_i * k.W - sv_x * dv[a];
      gx[a] += gd_x - gd_own;
      gv[a] += gdv_x - gdv_own;
    }
    pibar += mm * k.G * (uP + uPj);
    // d/d rho_i of j's terms, times rho_i^2 (divided once below).
    rsum += dvQj * mm * k.L + dvYj * m_i * k.W + sig_j * dvn * m_i * inv_re;
  });
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    gx[a] = lane_sum<kLanes>(gx[a]);
    gv[a] = lane_sum<kLanes>(gv[a]);
  }
  pibar = lane_sum<kLanes>(pibar);
  rsum = lane_sum<kLanes>(rsum);
  if (!live || q != 0) return;
  // pi_i = p_i / rho_i^2, p_i = k max(0, rho_i - rho0).
  const double rho_i = t.rho[i], p_i = t.p[i];
  const double inv_r2 = 1.0 / (rho_i * rho_i);
  const double pbar = pibar * inv_r2;
  double rbar = w.rbar[i] - rsum * inv_r2 - 2.0 * pibar * p_i * inv_r2 / rho_i;
  const double over = rho_i - c.rest;
  double kk = 0.0;
  if (over > 0.0) {
    rbar += pbar * c.stiff;
    kk = pbar * over;
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    w.gx[a][i] += gx[a];
    w.gv[a][i] += gv[a];
  }
  w.rbar_tot[i] = rbar;
  w.kk[i] = kk;
}

template <int kLanes>
__global__ void __launch_bounds__(kThreads) k_adj_density(StepConsts c, AdjTape t, AdjWork w) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = g / kLanes, q = g % kLanes;
  const bool live = i < c.n;
  const int ii = live ? i : 0;
  const size_t n = (size_t)c.n;
  const d4 xo = load_part(w, 0, n, ii);
  const double xi = xo.x, yi = xo.y, zi = xo.z;
  const double m_i = xo.w, rb_i = w.rbar_tot[ii];
  double gd[3] = {0.0, 0.0, 0.0};
  if (live) for_each_listed<kLanes>(c, t, i, q, xi, yi, zi, [&](int j) {
    // The forward's density test (p_i - p_j, world.rs:226-229); r = 0 pairs
    // (self, coincident particles) have W'(0) = 0.
    const d4 xj = load_part(w, 0, n, j);
    const double rb_j = w.rbar_tot[j];
    const double d[3] = {__dsub_rn(xi, xj.x), __dsub_rn(yi, xj.y), __dsub_rn(zi, xj.z)};
    const double r2 = norm2(d[0], d[1], d[2]);
    if (r2 > c.r2_guard) return;
    const double r = __dsqrt_rn(r2);
    if (!(r < c.h) || r <= 0.0 || r >= c.h0) return;
    const double qq = c.h0sq - r2;
    // W'(r) / r = -6 poly6_c (h0^2 - r^2)^2
    const double f = -6.0 * c.poly6_c * qq * qq * (xj.w * rb_i + m_i * rb_j);
#pragma unroll
    for (int a = 0; a < 3; ++a) gd[a] += f * d[a];
  });
#pragma unroll
  for (int a = 0; a < 3; ++a) gd[a] = lane_sum<kLanes>(gd[a]);
  if (!live || q != 0) return;
  const uint32_t ins = t.id[i];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    w.gx_ins[a][ins] = w.gx[a][i] + gd[a];
    w.gv_ins[a][ins] = w.gv[a][i];
  }
}

// acc[0] += sum a[0..n), acc[1] += sum b[0..n) in a fixed order: kSumBlocks
// blocks write partial sums, the last one to arrive adds them up (`arrived`
// ends at zero again).  One block took 17 us for 65,536 values.
constexpr int kSumThreads = 256;
__device__ __forceinline__ void block_sum2(double& x, double& y) {
  __shared__ double sa[kSumThreads], sb[kSumThreads];
  __syncthreads();
  sa[threadIdx.x] = x;
  sb[threadIdx.x] = y;
  __syncthreads();
  for (int o = kSumThreads / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sa[threadIdx.x] += sa[threadIdx.x + o];
      sb[threadIdx.x] += sb[threadIdx.x + o];
    }
    __syncthreads();
  }
  x = sa[0];
  y = sb[0];
}
__global__ void __launch_bounds__(kSumThreads) k_adj_sum2(int n, const double* __restrict__ a,
                                                          const double* __restrict__ b, double* acc, double* part,
                                                          unsigned* arrived) {
  __shared__ bool s_last;
  double x = 0.0, y = 0.0;
  for (int k = blockIdx.x * kSumThreads + threadIdx.x; k < n; k += kAdjSumBlocks * kSumThreads) {
    x += a[k];
    y += b[k];
  }
  block_sum2(x, y);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = x;
    part[2 * blockIdx.x + 1] = y;
    __threadfence();
    s_last = atomicAdd(arrived, 1u) == (unsigned)kAdjSumBlocks - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  x = y = 0.0;
  if (threadIdx.x < kAdjSumBlocks) {
    x = __ldcg(part + 2 * threadIdx.x);
    y = __ldcg(part + 2 * threadIdx.x + 1);
  }
  block_sum2(x, y);
  if (threadIdx.x == 0) {
    acc[0] += x;
    acc[1] += y;
    *arrived = 0;
  }
}

}  // namespace

void launch_adjoint_step(const StepConsts& c, const AdjTape& t, const AdjWork& w, cudaStream_t s) {
  if (c.n == 0) return;
  const int grid = (c.n + kThreads - 1) / kThreads;
  const int lanes = c.n < kLanesBelow ? 4 : 2;  // they share a warp
  const int pair_grid = (int)(((long long)c.n * lanes + kThreads - 1) / kThreads);
  k_adj_integrate<<<grid, kThreads, 0, s>>>(c, t, w);
  (lanes == 4 ? k_adj_force<4> : k_adj_force<2>)<<<pair_grid, kThreads, 0, s>>>(c, t, w);
  (lanes == 4 ? k_adj_density<4> : k_adj_density<2>)<<<pair_grid, kThreads, 0, s>>>(c, t, w);
  // param_acc = {d/d stiffness, d/d visc_k[0]}
  static_assert(kAdjSumBlocks <= kSumThreads, "one partial per thread");
  k_adj_sum2<<<kAdjSumBlocks, kSumThreads, 0, s>>>(c.n, w.kk, w.cc, w.param_acc, w.sum_part, w.sum_arrived);
}

}  // namespace phy
