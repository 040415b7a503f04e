// Nf=2 pseudofermion link force from a pair of solutions (X, Y), reference layout.
//
// Restates jaxqft/models/su3_wilson_nf2.py:1556-1576 per link (x, mu), with
// the boundary-phased link U = U_mu(x) (phase on x_mu = L_mu - 1):
//   c1_ac = sum_s conj(Y(x))_sa  [ (1 - g_mu) U X(x+mu) ]_sc
//   c2_dc = sum_s conj(U Y(x+mu))_sd [ (1 + g_mu) X(x) ]_sc
//   F_mu(x) = TA( transpose(c1 - c2) ),  TA(k) = (k - k^dag)/2 - tr/3
// (c2 follows from the reference's einsum "sa,st,ad,tc->dc" by moving U^dag
// onto Y(x+mu)).
//
// (1 -+ g_mu) has rank two and equals R R^dag with R^dag psi the two projected
// rows h_r(psi) of wl_hop.cuh (mu = 3: the stored rows carry a factor 2, so R R^dag
// is half their product).  Each spin sum is therefore a sum over two rows,
//   k_ca = sum_r (U h-_r(X(x+mu)))_c conj(h-_r(Y(x)))_a - h+_r(X(x))_c conj((U h+_r(Y(x+mu)))_a),
// and TA(k) needs only the three imaginary diagonals and three off-diagonal
// complex entries of k - k^dag: nine reals.
//
// Mapping: two threads per link, thread j forming row r = j of the four projections by
// the sector loads of ref_pair_kernel (wl_refsite.cuh); the links come from the gauge
// object's parity-split SoA copy; the nine reals of the pair are added by one xor-shuffle
// each.  The 64 links of a block are staged in shared memory and leave as one contiguous
// 9216-byte run.  Blocks of the four directions of the same sites are neighbours in the
// grid, so that a lattice of a few thousand sites still fills the GPU.
//
// The even-odd force f(K_oe X_e, -a Y_e) + f(X_e, -a K^dag_oe Y_e) (:1578-1597) is the same
// sum for the fields X_e + K_oe X_e and Y_e + K^dag_oe Y_e: a link joins an even and an odd
// site, and each of the two forces keeps the products in which its odd field meets the
// other's even one.  X[p] / Y[p] are therefore separate pointers per site parity.
//
// Bound by the latency of its loads at 16 warps per SM (128 registers): at 16^3x32 the L1 data
// pipe is 65 % busy, DRAM runs at 2.9 TB/s (178 MB for 1536 bytes per site, each link read and
// written once, each field once) and a warp waits for a load on 3 of 8 cycles between its
// instructions.  The kernel it replaced (one thread per link, AoS links and spinors in 16-byte
// loads 144 and 192 bytes apart, 186 registers) spent 80 % of the L1 pipe on those strides.
// Measured (B200): 2 x 12^3x24 force 102 -> 45 us (floor 20 us at the measured copy rate), even-odd force at
// 16^3x32, with its two hops, 368 -> 120 us (floor 27 us).
#pragma once
#include "wl_refsite.cuh"

namespace wl {

struct ForceArgs {
  Geom g;
  const double2* U;    // FP64 18-real links [p][mu][9][Vh]
  const double* X[2];  // field read at sites of parity p, [V][24] reals
  const double* Y[2];
  double2* F;          // [mu][V][3][3]
  double coef;
  int accumulate;
};

constexpr int kForceSites = 64;  // links per block (two threads each)

// nine reals of k - k^dag from one row: d[c] = Im k_cc, o[i] = (k - k^dag)_ab / 2 for ab = 01, 02, 12,
// with k_ca += w u_c conj(v_a)
WL_D void force_outer(const cplx<double> (&u)[3], const cplx<double> (&v)[3], double w, double (&d)[3],
                      cplx<double> (&o)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = fma(w, u[c].im * v[c].re - u[c].re * v[c].im, d[c]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int a = i == 2 ? 1 : 0, b = i == 0 ? 1 : 2;
    cplx<double> t = {0.0, 0.0};
    fmac_(t, v[b], u[a]);                              // u_a conj(v_b)
    t.re -= u[b].re * v[a].re + u[b].im * v[a].im;     // - conj(u_b) v_a
    t.im -= u[b].re * v[a].im - u[b].im * v[a].re;
    o[i].re = fma(0.5 * w, t.re, o[i].re);
    o[i].im = fma(0.5 * w, t.im, o[i].im);
  }
}

// uh = U h, times the boundary phase
template <int MU>
WL_D void force_transport(const Geom& g, const Link<double>& u, bool ph, const cplx<double> (&h)[3],
                          cplx<double> (&uh)[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    cplx<double> t = {0.0, 0.0};
#pragma unroll
    for (int b = 0; b < 3; ++b) fma_(t, u.m[a][b], h[b]);
    uh[a] = ph ? t * cplx<double>{g.ph_re[MU], g.ph_im[MU]} : t;
  }
}

template <int MU, int W, bool SECT>
WL_D void force_link(const ForceArgs& A, const Site& s, int parity, size_t flat, int j, unsigned pm, double (&d)[3],
                     cplx<double> (&o)[3]) {
  const Geom& g = A.g;
  const double sg = 1.0 - 2.0 * j;
  const int nb = neighbor(g, s, MU, +1);
  int tn = s.x[3];
  if (MU == 3) tn = tn == g.L[3] - 1 ? 0 : tn + 1;
  const size_t fn = (size_t)(2 * nb + ((MU == 3 ? tn : s.x[3]) & 1)) * 24;
  const size_t fx = flat * 24;
  const bool ph = g.ph_on[MU] && s.x[MU] == g.L[MU] - 1;
  constexpr double w = MU == 3 ? 0.5 : 1.0;
  Link<double> u;
  ld_link(A.U, (unsigned)g.Vh, parity, MU, s.c, u);
  cplx<double> h[3], v[3], t[3];
  refpair_project<MU, -1, W, SECT>(A.X[1 - parity] + fn, j, sg, pm, h);
  refpair_project<MU, -1, W, SECT>(A.Y[parity] + fx, j, sg, pm, v);
  force_transport<MU>(g, u, ph, h, t);
  force_outer(t, v, w, d, o);
  refpair_project<MU, +1, W, SECT>(A.Y[1 - parity] + fn, j, sg, pm, h);
  refpair_project<MU, +1, W, SECT>(A.X[parity] + fx, j, sg, pm, v);
  force_transport<MU>(g, u, ph, h, t);
  force_outer(v, t, -w, d, o);
}

template <int W, bool SECT>
__global__ void __launch_bounds__(2 * kForceSites, 4) pf_force_kernel(ForceArgs A) {
  __shared__ double2 sm[kForceSites * 9];
  const Geom& g = A.g;
  const int mu = blockIdx.x & 3;
  const int f0 = (int)(blockIdx.x >> 2) * kForceSites;
  const int i = threadIdx.x >> 1, j = threadIdx.x & 1;
  const bool act = f0 + i < g.V;
  const unsigned pm = __ballot_sync(0xffffffffu, act);  // both threads of a pair share `act`
  if (act) {
    const Site s = site_of_flat(g, f0 + i);
    const int parity = (s.x[0] + s.x[1] + s.x[2] + s.x[3]) & 1;
    double d[3] = {0.0, 0.0, 0.0};
    cplx<double> o[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    switch (mu) {
      case 0: force_link<0, W, SECT>(A, s, parity, (size_t)(f0 + i), j, pm, d, o); break;
      case 1: force_link<1, W, SECT>(A, s, parity, (size_t)(f0 + i), j, pm, d, o); break;
      case 2: force_link<2, W, SECT>(A, s, parity, (size_t)(f0 + i), j, pm, d, o); break;
      default: force_link<3, W, SECT>(A, s, parity, (size_t)(f0 + i), j, pm, d, o); break;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      d[c] = A.coef * (d[c] + __shfl_xor_sync(pm, d[c], 1));
      o[c].re = A.coef * (o[c].re + __shfl_xor_sync(pm, o[c].re, 1));
      o[c].im = A.coef * (o[c].im + __shfl_xor_sync(pm, o[c].im, 1));
    }
    const double tr = (d[0] + d[1] + d[2]) / 3.0;
    double2* q = sm + i * 9;
    if (j == 0) {  // upper triangle and the first diagonal entry
      q[0] = make_double2(0.0, d[0] - tr);
      q[1] = make_double2(o[0].re, o[0].im);
      q[2] = make_double2(o[1].re, o[1].im);
      q[5] = make_double2(o[2].re, o[2].im);
    } else {
      q[3] = make_double2(-o[0].re, o[0].im);
      q[4] = make_double2(0.0, d[1] - tr);
      q[6] = make_double2(-o[1].re, o[1].im);
      q[7] = make_double2(-o[2].re, o[2].im);
      q[8] = make_double2(0.0, d[2] - tr);
    }
  }
  __syncthreads();
  const int n = 9 * min(kForceSites, g.V - f0);
  double2* F = A.F + ((size_t)mu * g.V + f0) * 9;
  for (int k = threadIdx.x; k < n; k += 2 * kForceSites) {
    double2 v = sm[k];
    if (A.accumulate) {
      const double2 old = F[k];
      v.x += old.x;
      v.y += old.y;
    }
    F[k] = v;
  }
}

}  // namespace wl
