// Pure-gauge pieces of the SU(3) HMC on the device, reference layout BMXYIJ
// (links [B][mu][Lx][Ly][Lz][Lt][3][3] complex128, t fastest, periodic):
//   * Wilson plaquette sum  sum_{x, mu<nu} Re Tr U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag
//     (jaxqft/models/su3_ym.py:274-286 action_reference, 369-388 average_plaquette)
//   * gauge force  F_mu(x) = -(beta/3) TA(U_mu(x) V_mu(x)^dag) with the staple
//     V_mu(x) = sum_{nu != mu} U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu)
//     (su3_ym.py:298-327 _staple / force_reference)
//   * exponential drift  U <- exp(dt P) U  (su3_ym.py:349-350 evolve_q_reference with
//     exp_method "expm", su3_ym.py:265-272)
//   * kinetic term  -1/2 sum Re Tr P P  (su3_ym.py:362-364)
// All FP64.  One thread per link (force, drift, kinetic) or per site (plaquette);
// sums are deterministic block partials finished by reduce_finalize_kernel.
#pragma once
#include "wl_refsite.cuh"

namespace wl {

struct M3 {
  cplx<double> m[3][3];
};

WL_D void m3_load(M3& a, const double2* p) {
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = ldg(p + k);
    a.m[k / 3][k % 3] = {v.x, v.y};
  }
}

// c = a b ; c = a b^dag ; c = a^dag b
WL_D void m3_mul(const M3& a, const M3& b, M3& c) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx<double> s = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) fma_(s, a.m[i][k], b.m[k][j]);
      c.m[i][j] = s;
    }
}
WL_D void m3_mul_nd(const M3& a, const M3& b, M3& c) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx<double> s = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) fmac_(s, b.m[j][k], a.m[i][k]);  // a_ik conj(b_jk)
      c.m[i][j] = s;
    }
}
WL_D void m3_mul_dn(const M3& a, const M3& b, M3& c) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx<double> s = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) fmac_(s, a.m[k][i], b.m[k][j]);  // conj(a_ki) b_kj
      c.m[i][j] = s;
    }
}

// Re Tr(a b^dag) = sum_ij Re(a_ij conj(b_ij))
WL_D double m3_retr_nd(const M3& a, const M3& b) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) s += a.m[i][j].re * b.m[i][j].re + a.m[i][j].im * b.m[i][j].im;
  return s;
}

// TA(x) = (x - x^dag)/2 - Tr(x - x^dag)/6 * 1   (su3_ym.py:56-67)
WL_D void m3_ta(const M3& x, M3& y, double coef) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      y.m[i][j] = {0.5 * (x.m[i][j].re - x.m[j][i].re), 0.5 * (x.m[i][j].im + x.m[j][i].im)};
  const double tr = (y.m[0][0].im + y.m[1][1].im + y.m[2][2].im) / 3.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) y.m[i][i].im -= tr;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) y.m[i][j] = coef * y.m[i][j];
}

// exp(A): the degree-18 Taylor polynomial of a = A 2^-s (max-row-sum norm <= 1, truncation 1/19! ~ 8e-18),
// squared s times (scaling and squaring, as in Moler and Van Loan, "Nineteen dubious ways to compute the
// exponential of a matrix", method 3).  The polynomial is evaluated modulo the characteristic polynomial: by
// Cayley-Hamilton a^3 = t a^2 - m a + d with t = tr a, m = (t^2 - tr a^2) / 2, d = det a, so Horner's rule runs
// on the three coefficients of q0 + q1 a + q2 a^2 (12 FMAs a step) and one matrix product, a^2, is all that is
// left of the fourteen products of a matrix Horner scheme.
WL_D void m3_exp(const M3& A, M3& E) {
  double nrm = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double r = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) r += fabs(A.m[i][j].re) + fabs(A.m[i][j].im);
    nrm = fmax(nrm, r);
  }
  int s = 0;
  while (nrm > 1.0 && s < 64) {  // bounded: at most 64 halvings
    nrm *= 0.5;
    ++s;
  }
  const double sc = ldexp(1.0, -s);
  M3 a, a2;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) a.m[i][j] = sc * A.m[i][j];
  m3_mul(a, a, a2);
  const cplx<double> t = a.m[0][0] + a.m[1][1] + a.m[2][2];
  const cplx<double> m = 0.5 * (t * t - (a2.m[0][0] + a2.m[1][1] + a2.m[2][2]));
  const cplx<double> d = a.m[0][0] * (a.m[1][1] * a.m[2][2] - a.m[1][2] * a.m[2][1]) -
                         a.m[0][1] * (a.m[1][0] * a.m[2][2] - a.m[1][2] * a.m[2][0]) +
                         a.m[0][2] * (a.m[1][0] * a.m[2][1] - a.m[1][1] * a.m[2][0]);
  // 1/k!, k = 0..18 (exact quotients rounded by the compiler)
  constexpr double c[19] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320,
                            1.0 / 362880, 1.0 / 3628800, 1.0 / 39916800, 1.0 / 479001600, 1.0 / 6227020800.0,
                            1.0 / 87178291200.0, 1.0 / 1307674368000.0, 1.0 / 20922789888000.0,
                            1.0 / 355687428096000.0, 1.0 / 6402373705728000.0};
  cplx<double> q0 = {c[18], 0.0}, q1 = {0.0, 0.0}, q2 = {0.0, 0.0};
#pragma unroll
  for (int k = 17; k >= 0; --k) {  // (q0 + q1 a + q2 a^2) a + c_k
    const cplx<double> p0 = q2 * d, p1 = q2 * m, p2 = q2 * t;
    q2 = q1 + p2;
    q1 = q0 - p1;
    q0 = {c[k] + p0.re, p0.im};
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx<double> e = {0.0, 0.0};
      fma_(e, q2, a2.m[i][j]);
      fma_(e, q1, a.m[i][j]);
      E.m[i][j] = i == j ? e + q0 : e;
    }
  if (s > 0) {
    M3 w;
#pragma unroll 1
    for (int q = 0; q < s; ++q) {
      m3_mul(E, E, w);
      E = w;
    }
  }
}

struct GaugeArgs {
  Geom g;
  const double2* U;  // [B][4][V][9]
  const double2* P;  // [B][4][V][9] (drift, kinetic)
  double2* out;      // [B][4][V][9]
  int batch;
  double coef;       // force: -beta/3 ; drift: dt
  double* partials;  // [batch][nblk]
};

WL_D long long gflat(const Geom& g, int x0, int x1, int x2, int x3) {
  return (((long long)x0 * g.L[1] + x1) * g.L[2] + x2) * g.L[3] + x3;
}

WL_D void gcoords(const Geom& g, long long f, int (&x)[4]) {
  x[3] = (int)(f % g.L[3]);
  f /= g.L[3];
  x[2] = (int)(f % g.L[2]);
  f /= g.L[2];
  x[1] = (int)(f % g.L[1]);
  x[0] = (int)(f / g.L[1]);
}

WL_D long long gshift(const Geom& g, const int (&x)[4], int mu, int dmu, int nu, int dnu) {
  int y[4] = {x[0], x[1], x[2], x[3]};
  y[mu] += dmu;
  y[nu] += dnu;
#pragma unroll
  for (int d = 0; d < 4; ++d) y[d] = y[d] < 0 ? y[d] + g.L[d] : (y[d] >= g.L[d] ? y[d] - g.L[d] : y[d]);
  return gflat(g, y[0], y[1], y[2], y[3]);
}

WL_D const double2* glink(const GaugeArgs& A, const double2* base, int b, int mu, long long f) {
  return base + (((long long)b * 4 + mu) * A.g.V + f) * 9;
}

// 16-byte asynchronous copy global -> shared, and the wait for all of this thread's copies
WL_D void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
WL_D void cp16_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

WL_D void m3_lds(M3& a, const double2* p) {
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = p[k];
    a.m[k / 3][k % 3] = {v.x, v.y};
  }
}

// ---------------------------------------------------------------- force
// One thread per link.  A block is 32 consecutive sites with one warp per direction, so that the 76 link reads of a
// site (31 distinct ones per row) meet in L1; the 32 results of a warp are staged in shared memory and leave as one
// contiguous 4608-byte run.  Bound by the L1 data pipe: the reads are 144-byte matrices in 16-byte loads, which keep it
// 86 % busy at 16^3x32 (60 % of their sectors hit), next to 1404 FP64 FMAs a link (FP64 pipe 40 %).  162 registers
// (three matrices and the staple sum live) leave 12 warps per SM.
// Measured (B200, us of the force alone, three prepared configurations in turn) against blocks of 128 sites of one
// direction with unstaged stores: 8^4 10.3 -> 10.3 (the host's share), 12^3x24 55.5 -> 53.4, 16^3x32 174 -> 157
// (floor 24 us of DRAM, 40 us of FP64), three configurations of 16^3x32 515 -> 458.  Also measured and not kept: the
// links copied first to a matrix-element-major scratch, whose reads are contiguous (15.4, 55.1, 159, 469 us: the copy
// takes what the reads save); the 31 rows of a 16-site segment staged in shared memory with 18 threads a site; 4D site
// tiles per block.
// grid: x over groups of 32 sites, z = batch
__global__ void __launch_bounds__(128, 3) gauge_force_kernel(GaugeArgs A) {
  __shared__ double2 sm[4][32 * 9];
  const Geom& g = A.g;
  const int mu = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f0 = (int)blockIdx.x * 32, f = f0 + lane;
  const size_t plane = (size_t)blockIdx.z * 4;
  if (f < g.V) {
    const double2* links = A.U + plane * 9 * g.V;
    const Site s = site_of_flat(g, f);
    const auto load = [&](M3& a, int dir, int site) { m3_load(a, links + ((size_t)dir * g.V + site) * 9); };
    const auto at = [&](int mu1, int d1, int mu2, int d2) { return (int)gshift(g, s.x, mu1, d1, mu2, d2); };
    M3 st, t, u, v;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) st.m[i][j] = {0.0, 0.0};
#pragma unroll 1
    for (int n = 1; n < 4; ++n) {
      const int nu = (mu + n) & 3;
      // forward: U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag
      load(u, nu, f);
      load(v, mu, at(nu, +1, mu, 0));
      m3_mul(u, v, t);
      load(u, nu, at(mu, +1, nu, 0));
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int k = 0; k < 3; ++k) fmac_(st.m[i][j], u.m[j][k], t.m[i][k]);
      // backward: U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu)
      const int fm = at(nu, -1, mu, 0);
      load(u, nu, fm);
      load(v, mu, fm);
      m3_mul_dn(u, v, t);
      load(u, nu, at(nu, -1, mu, +1));
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int k = 0; k < 3; ++k) fma_(st.m[i][j], t.m[i][k], u.m[k][j]);
    }
    load(u, mu, f);
    m3_mul_nd(u, st, t);  // U_mu(x) V^dag
    m3_ta(t, v, A.coef);
#pragma unroll
    for (int k = 0; k < 9; ++k) sm[mu][lane * 9 + k] = make_double2(v.m[k / 3][k % 3].re, v.m[k / 3][k % 3].im);
  }
  __syncwarp();
  double2* out = A.out + ((plane + mu) * g.V + f0) * 9;
  for (int q = lane; q < 9 * min(32, g.V - f0); q += 32) out[q] = sm[mu][q];
}

// ---------------------------------------------------------------- drift
// out = exp(coef * P) U, one thread per link (grid.x over all B*4*V links).  A warp copies the P and U of its 32
// links to shared memory as two contiguous 4608-byte runs, works from there (144-byte rows: no bank conflicts) and
// returns the result the same way.  Bound by DRAM (432 bytes a link) next to FP64 arithmetic (about 560 FMAs).
// The kernel it replaced evaluated a degree-14 matrix Horner scheme (about 2450 FMAs) on 16-byte accesses 144 bytes
// apart.  Measured at 16^3x32: 95 -> 38 us (226 MB: 35 us at the measured copy rate); 3, 4 or 5 blocks per SM alike.
constexpr int kEvolveThreads = 128;

__global__ void __launch_bounds__(kEvolveThreads, 4) gauge_evolve_kernel(GaugeArgs A) {
  __shared__ double2 sm[kEvolveThreads / 32][2][32 * 9];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long l0 = ((long long)blockIdx.x * (kEvolveThreads / 32) + warp) * 32;
  const long long total = (long long)A.batch * 4 * A.g.V;
  if (l0 >= total) return;  // uniform per warp; only warp barriers below
  const int n = (int)min(32LL, total - l0);
  for (int q = lane; q < n * 9; q += 32) {
    cp16(&sm[warp][0][q], A.P + l0 * 9 + q);
    cp16(&sm[warp][1][q], A.U + l0 * 9 + q);
  }
  cp16_wait();
  __syncwarp();
  if (lane < n) {
    M3 p, e;
    m3_lds(p, &sm[warp][0][lane * 9]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) p.m[i][j] = A.coef * p.m[i][j];
    m3_exp(p, e);
    m3_lds(p, &sm[warp][1][lane * 9]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        cplx<double> r = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 3; ++k) fma_(r, e.m[i][k], p.m[k][j]);
        sm[warp][0][lane * 9 + i * 3 + j] = make_double2(r.re, r.im);
      }
  }
  __syncwarp();
  for (int q = lane; q < n * 9; q += 32) A.out[l0 * 9 + q] = sm[warp][0][q];
}

// per-site plaquette sums (grid: x over sites, z = batch); partials[b][block]
__global__ void __launch_bounds__(128) gauge_plaquette_kernel(GaugeArgs A) {
  __shared__ double sm[32];
  const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.z;
  double v[1] = {0.0};
  if (f < A.g.V) {
    int x[4];
    gcoords(A.g, f, x);
    M3 um, un, a, c, t;
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
      m3_load(um, glink(A, A.U, b, mu, f));
#pragma unroll 1
      for (int nu = mu + 1; nu < 4; ++nu) {
        // Re Tr (U_mu(x) U_nu(x+mu)) (U_nu(x) U_mu(x+nu))^dag
        m3_load(t, glink(A, A.U, b, nu, gshift(A.g, x, mu, +1, nu, 0)));
        m3_mul(um, t, a);
        m3_load(un, glink(A, A.U, b, nu, f));
        m3_load(t, glink(A, A.U, b, mu, gshift(A.g, x, nu, +1, mu, 0)));
        m3_mul(un, t, c);
        v[0] += m3_retr_nd(a, c);
      }
    }
  }
  block_sum<1>(v, sm);
  if (threadIdx.x == 0) A.partials[(long long)b * gridDim.x + blockIdx.x] = v[0];
}

// -1/2 Re Tr P P per link (grid: x over links of one configuration, z = batch)
__global__ void __launch_bounds__(128) gauge_kinetic_kernel(GaugeArgs A) {
  __shared__ double sm[32];
  const long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.z;
  double v[1] = {0.0};
  if (l < 4LL * A.g.V) {
    M3 p;
    m3_load(p, A.P + ((long long)b * 4 * A.g.V + l) * 9);
    double s = 0.0;  // Re Tr P P = sum_ij Re(p_ij p_ji)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) s += p.m[i][j].re * p.m[j][i].re - p.m[i][j].im * p.m[j][i].im;
    v[0] = -0.5 * s;
  }
  block_sum<1>(v, sm);
  if (threadIdx.x == 0) A.partials[(long long)b * gridDim.x + blockIdx.x] = v[0];
}

}  // namespace wl
