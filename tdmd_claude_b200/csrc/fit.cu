// fit.cu -- force-matching loss over a set of snapshots and its gradient
// with respect to the potential's parameters, by the adjoint of the force
// expressions (tdmd_fit_* in the C ABI).
//
// No reference counterpart: tdmd_Claude computes no gradients.  The forces
// are the ones of its Morse (src/potentials/morse.hpp:37-55) and EAM
// (src/potentials/eam_alloy.cpp:196-295) paths; the loss is
//   L = 1/(3 M) sum_i |F_i - T_i|^2   over all M atoms of all snapshots.
// With G_i = dL/dF_i = 2 (F_i - T_i) / (3 M) and, for an ordered pair (i, j)
// of the full neighbor list, d = r_i - r_j and q_ij = G_i . d / r:
//   Morse  F_i = sum_j f(r) d,  dL/dtheta = sum_(i,j) (G_i . d) df/dtheta;
//   EAM    f = -(phi'_p + F'_i rho'_tj + F'_j rho'_ti) / r, and
//     phi_p coefficients:   -q_ij * dphi'/dc            at r
//     rho_tj coefficients:  -q_ij F'_i drho'/dc          at r
//     rho_ti coefficients:  -q_ij F'_j drho'/dc          at r
//     F_ti coefficients:    w_i * dF'/dc                 at rho_i
//     rho_tj coefficients:  w_i F''_i * drho/dc          at r
//   with the adjoint density weight
//     w_i = -sum_j rho'_tj(r) (G_i - G_j) . d / r.
// No second derivative in positions is needed: the parameters enter the
// forces directly, and through F'(rho) the embedding's second derivative.
//
// B200 layout: the snapshots are batched replicas of one box (one launch per
// pass over all of them), neighbor lists are built once at creation, and
// every pass works on device arrays only (parameters, coefficients, loss and
// gradients are device pointers), so a fitting loop needs no host round trip
// per step.  Gradients accumulate in FP64 (per-block partials for the three
// Morse parameters; FP64 atomics into the coefficient arrays for EAM).
// Passes: Morse = forces+G, gradient; EAM = density (+F', F''), forces+G,
// adjoint weights w_i (+ F terms), then the phi and rho terms over the
// unordered pairs.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <optional>
#include <vector>

#include "buffers.cuh"
#include "common.cuh"
#include "forces.cuh"
#include "launch.cuh"
#include "replica_geo.cuh"
#include "replicas.cuh"

namespace tdmd_b200 {
namespace {

constexpr int kThreads = 256;
constexpr int kPart = 4;  // doubles per block partial

// One row (a, b, c, d) per spline interval, so that a pair's lookup is one
// 32-byte load per spline (the packed a|b|c|d arrays the caller passes take
// four 8-byte gathers: 33 L1 cycles for a warp's random intervals, 19 for one
// row).
template <class T>
__device__ __forceinline__ T row_value(const double4& r, T dx) {
  const T a = static_cast<T>(r.x), b = static_cast<T>(r.y), c = static_cast<T>(r.z),
          d = static_cast<T>(r.w);
  return a + dx * (b + dx * (c + dx * d));
}
template <class T>
__device__ __forceinline__ T row_deriv(const double4& r, T dx) {
  const T b = static_cast<T>(r.y), c = static_cast<T>(r.z), d = static_cast<T>(r.w);
  return b + dx * (T(2) * c + T(3) * d * dx);
}

// Gradient of an interval's coefficients in a packed a|b|c|d array: wd times
// the derivative's basis (0, 1, 2x, 3x^2) plus wv times the value's
// (1, x, x^2, x^3).
__device__ __forceinline__ void add_deriv_basis(double* g, int ns, int k, double dx, double wd) {
  atomicAdd(g + ns + k, wd);
  atomicAdd(g + 2 * ns + k, 2.0 * wd * dx);
  atomicAdd(g + 3 * ns + k, 3.0 * wd * dx * dx);
}
__device__ __forceinline__ void add_both_bases(double* g, int ns, int k, double dx, double wd,
                                               double wv) {
  atomicAdd(g + k, wv);
  atomicAdd(g + ns + k, fma(wv, dx, wd));
  atomicAdd(g + 2 * ns + k, dx * fma(wv, dx, 2.0 * wd));
  atomicAdd(g + 3 * ns + k, dx * dx * fma(wv, dx, 3.0 * wd));
}

__device__ __forceinline__ int pair_index(int ti, int tj, int nt) {
  if (ti > tj) {
    const int t = ti;
    ti = tj;
    tj = t;
  }
  return ti * nt - ti * (ti + 1) / 2 + tj;
}

unsigned high_word(double x) {
  unsigned long long u;
  std::memcpy(&u, &x, sizeof u);
  return static_cast<unsigned>(u >> 32);
}

// Device view of the EAM coefficient arrays being fitted, the row copies the
// passes read and the gradients (types 0-based here).
struct FitEam {
  const double* F;
  const double4* rows;  // [nt + npairs][nsr]: rho_t, then phi_p
  double* gF;
  double* grho;
  double* gphi;
  int nt, nsf, nsr;
  double drho, dr, inv_dr;
  unsigned in_lo, in_span;
  __device__ __forceinline__ double4 rho_row(int t, int k) const {
    return ld_d4(rows + static_cast<long long>(t) * nsr + k);
  }
  __device__ __forceinline__ double4 phi_row(int p, int k) const {
    return ld_d4(rows + static_cast<long long>(nt + p) * nsr + k);
  }
  // The interval int(r / dr) and the offset in it.  Each interval's
  // coefficients are free parameters here: a pair on a knot must go where the
  // division puts it, because the neighboring cubic may differ in value and
  // slope and owns another part of the gradient.  So the product with 1/dr (as
  // in spline_idx_mul) decides only offsets inside (in_lo, in_lo + in_span) of
  // the high word; the others (about two in a million of thermal distances,
  // whole shells of an ideal lattice, and what needs the clamp) take the
  // quotient as the division rounds it: two Newton corrections of r * (1/dr)
  // with exact remainders (Markstein's theorem).
  __device__ __forceinline__ int seg(double r, double& dx) const {
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
    const double z = fma(r, inv_dr, -0.5) + kRound;
    int k = __double2loint(z);
    dx = fma(-(z - kRound), dr, r);
    if (static_cast<unsigned>(__double2hiint(dx)) - in_lo >= in_span) {
      double q = r * inv_dr;
      q = fma(fma(-q, dr, r), inv_dr, q);
      q = fma(fma(-q, dr, r), inv_dr, q);
      k = min(static_cast<int>(q), nsr - 1);
      dx = fma(-static_cast<double>(k), dr, r);
    }
    return k;
  }
};

// x / r, rounded once.
__device__ __forceinline__ double over_radius(double x, double r, double rinv) {
  return div_r(x, r, rinv);
}
__device__ __forceinline__ double over_radius(double x, float r, float /*rinv*/) {
  return x / static_cast<double>(r);
}

// Block partial sums: lane merge -> warp -> block; thread 0 writes kPart.
template <int NV>
__device__ __forceinline__ void write_partials(double (&v)[NV], double* part) {
  __shared__ double red[32 * NV];
  block_sum<NV>(v, red);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) part[static_cast<long long>(blockIdx.x) * kPart + k] = v[k];
  }
}

template <class T, int LPA>
__device__ __forceinline__ T lane_sum(T v) {
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}

// Atom i's share of the loss; G_i = dL/dF_i goes out with w in the record's
// fourth word.
__device__ __forceinline__ double residual(double fx, double fy, double fz,
                                           const double* __restrict__ target, double c, int i,
                                           double w, double4* __restrict__ G,
                                           double* __restrict__ fout) {
  const double ex = fx - target[3ll * i], ey = fy - target[3ll * i + 1],
               ez = fz - target[3ll * i + 2];
  G[i] = make_double4(2.0 * c * ex, 2.0 * c * ey, 2.0 * c * ez, w);
  if (fout) {
    fout[3ll * i] = fx;
    fout[3ll * i + 1] = fy;
    fout[3ll * i + 2] = fz;
  }
  double v = c * ex * ex;
  v += c * ey * ey;
  v += c * ez * ez;
  return v;
}

// ---------------------------------------------------------------------------
// Morse
// ---------------------------------------------------------------------------
template <class Geo, int LPA>
__global__ void __launch_bounds__(kThreads) k_fm_morse_force(
    Geo g, NbrView nl, int n, const double* __restrict__ prm, double rc_sq,
    const double* __restrict__ target, double c, double4* __restrict__ G,
    double* __restrict__ fout, double* __restrict__ part) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA, sub = tid % LPA;
  const bool active = i < n;
  const T D = static_cast<T>(prm[0]), alpha = static_cast<T>(prm[1]);
  const double r0d = prm[2];
  Acc<T> fx, fy, fz;
  if (active) {
    const typename Geo::Own o = g.own(i);
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      typename Geo::Pair pr;
      g.pair(o, __ldg(nl.nbr + row + k), pr);
      if (pr.r2 < static_cast<T>(rc_sq)) {
        T r, rinv;
        double rd;
        g.radius(o, pr, r, rinv, rd);
        const T ex = exp(-alpha * static_cast<T>(rd - r0d));
        const T fpair = -div_r(T(2) * D * alpha * (T(1) - ex) * ex, r, rinv);
        fx.add(mul_rn(fpair, pr.dx));
        fy.add(mul_rn(fpair, pr.dy));
        fz.add(mul_rn(fpair, pr.dz));
      }
    }
  }
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) {
    fx.shfl_merge(s);
    fy.shfl_merge(s);
    fz.shfl_merge(s);
  }
  double v[1] = {0.0};
  if (active && sub == 0) {
    v[0] = residual(fx.value(), fy.value(), fz.value(), target, c, i, 0.0, G, fout);
  }
  write_partials<1>(v, part);
}

template <class Geo, int LPA>
__global__ void __launch_bounds__(kThreads) k_fm_morse_grad(Geo g, NbrView nl, int n,
                                                            const double* __restrict__ prm,
                                                            double rc_sq,
                                                            const double4* __restrict__ G,
                                                            double* __restrict__ part) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA, sub = tid % LPA;
  const double D = prm[0], alpha = prm[1], r0 = prm[2];
  const T Dt = static_cast<T>(D), at = static_cast<T>(alpha);
  double v[3] = {0.0, 0.0, 0.0};
  if (i < n) {
    const typename Geo::Own o = g.own(i);
    const double4 gi = G[i];
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      typename Geo::Pair pr;
      g.pair(o, __ldg(nl.nbr + row + k), pr);
      if (pr.r2 < static_cast<T>(rc_sq)) {
        T r, rinv;
        double rd;
        g.radius(o, pr, r, rinv, rd);
        const T ex = exp(-at * static_cast<T>(rd - r0));
        const T ome = T(1) - ex;
        const double gd = over_radius(gi.x * static_cast<double>(pr.dx) +
                                          gi.y * static_cast<double>(pr.dy) +
                                          gi.z * static_cast<double>(pr.dz),
                                      r, rinv);
        // df/dtheta * r (the 1/r is folded into gd)
        const T dD = -T(2) * at * ome * ex;
        const T da = -T(2) * Dt * (ome * ex - at * (T(1) - T(2) * ex) *
                                               static_cast<T>(rd - r0) * ex);
        const T dr0 = -T(2) * Dt * at * at * (T(1) - T(2) * ex) * ex;
        v[0] += gd * static_cast<double>(dD);
        v[1] += gd * static_cast<double>(da);
        v[2] += gd * static_cast<double>(dr0);
      }
    }
  }
  write_partials<3>(v, part);
}

// Sums nblk block partials (kPart doubles each) in block order:
// out[0..nv) = column sums; a second block does the same for part2 / out2.
__global__ void k_fm_sum(const double* __restrict__ part, int nv, double* __restrict__ out,
                         const double* __restrict__ part2, int nv2, double* __restrict__ out2,
                         int nblk) {
  dependent_launch_prologue();
  if (blockIdx.x == 1) {
    part = part2;
    nv = nv2;
    out = out2;
  }
  __shared__ double red[32 * kPart];
  double v[kPart] = {0.0, 0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < nblk; b += blockDim.x)
    for (int k = 0; k < nv; ++k) v[k] += part[static_cast<long long>(b) * kPart + k];
  block_sum<kPart>(v, red);
  if (threadIdx.x == 0)
    for (int k = 0; k < nv; ++k) out[k] = v[k];
}

// ---------------------------------------------------------------------------
// EAM
// ---------------------------------------------------------------------------
// Row copies of the r splines and zeroed gradients, before the passes.
__global__ void k_fm_rows(const double* __restrict__ rho, const double* __restrict__ phi, int nt,
                          int np, int nsr, double4* __restrict__ rows, double* __restrict__ gF,
                          long long nF, double* __restrict__ grho, double* __restrict__ gphi) {
  dependent_launch_prologue();
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long nr = static_cast<long long>(nt) * nsr, n = nr + static_cast<long long>(np) * nsr;
  for (long long q = tid; q < n; q += step) {
    const long long w = q < nr ? q : q - nr;  // within rho or phi
    const double* c = (q < nr ? rho : phi) + 4 * nsr * (w / nsr) + w % nsr;
    rows[q] = make_double4(c[0], c[nsr], c[2 * nsr], c[3 * nsr]);
  }
  if (!gF) return;
  for (long long q = tid; q < nF; q += step) gF[q] = 0.0;
  for (long long q = tid; q < 4 * nr; q += step) grho[q] = 0.0;
  for (long long q = tid; q < 4 * (n - nr); q += step) gphi[q] = 0.0;
}

// rho_i, then F' and F''; the force pass's gather records {position, F'}.
template <class Geo, int LPA>
__global__ void __launch_bounds__(kThreads) k_fm_eam_density(
    Geo g, NbrView nl, int n, const int* __restrict__ types, FitEam e, double rc_sq,
    double* __restrict__ rho_out, double* __restrict__ fp_out, double* __restrict__ fpp_out,
    double4* __restrict__ rec_d, int4* __restrict__ rec_q) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA, sub = tid % LPA;
  const bool active = i < n;
  const bool multi = e.nt > 1;
  Acc<T> rho;
  typename Geo::Own o{};
  if (active) {
    o = g.own(i);
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      const int j = __ldg(nl.nbr + row + k);
      typename Geo::Pair pr;
      g.pair(o, j, pr);
      if (pr.r2 < static_cast<T>(rc_sq)) {
        T r, rinv;
        double rd;
        g.radius(o, pr, r, rinv, rd);
        double dx;
        const int kk = e.seg(rd, dx);
        const int tj = multi ? __ldg(types + j) - 1 : 0;
        rho.add(row_value<T>(e.rho_row(tj, kk), static_cast<T>(dx)));
      }
    }
  }
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) rho.shfl_merge(s);
  if (active && sub == 0) {
    const double rh = rho.value();
    const double* F = e.F + 4ll * e.nsf * (multi ? __ldg(types + i) - 1 : 0);
    double dx;
    const int kk = spline_idx(rh, e.drho, e.nsf + 1, dx);
    const double b = __ldg(F + e.nsf + kk), c = __ldg(F + 2 * e.nsf + kk),
                 d = __ldg(F + 3 * e.nsf + kk);
    const double fp = b + dx * (2.0 * c + 3.0 * d * dx);
    rho_out[i] = rh;
    fp_out[i] = fp;
    fpp_out[i] = 2.0 * c + 6.0 * d * dx;
    if constexpr (Geo::kRecords) {
      int4 rec = g.record(o);
      rec.w = __float_as_int(static_cast<float>(fp));
      rec_q[i] = rec;
    } else {
      rec_d[i] = make_double4(o.x, o.y, o.z, fp);
    }
  }
}

// Forces from the {position, F'} records, residuals, G.
template <class Geo, int LPA>
__global__ void __launch_bounds__(kThreads) k_fm_eam_force(
    Geo g, NbrView nl, int n, const int* __restrict__ types, FitEam e, double rc_sq,
    const double* __restrict__ fp, const double* __restrict__ target, double c,
    double4* __restrict__ G, double* __restrict__ fout, double* __restrict__ part) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA, sub = tid % LPA;
  const bool active = i < n;
  const bool multi = e.nt > 1;
  Acc<T> fx, fy, fz;
  if (active) {
    const typename Geo::Own o = g.own(i);
    const int ti = multi ? __ldg(types + i) - 1 : 0;
    const T fpi = static_cast<T>(fp[i]);
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      const int j = __ldg(nl.nbr + row + k);
      typename Geo::Pair pr;
      g.pair(o, j, pr);
      if (pr.r2 < static_cast<T>(rc_sq)) {
        T r, rinv;
        double rd;
        g.radius(o, pr, r, rinv, rd);
        const int tj = multi ? __ldg(types + j) - 1 : 0;
        double dxd;
        const int kk = e.seg(rd, dxd);
        const T dx = static_cast<T>(dxd);
        const T dphi = row_deriv<T>(e.phi_row(multi ? pair_index(ti, tj, e.nt) : 0, kk), dx);
        const T drj = row_deriv<T>(e.rho_row(tj, kk), dx);
        const T dri = ti == tj ? drj : row_deriv<T>(e.rho_row(ti, kk), dx);
        const T fpj = static_cast<T>(g.gather_fp(pr, 0));
        const T fpair = -div_r(dphi + fpi * drj + fpj * dri, r, rinv);
        fx.add(mul_rn(fpair, pr.dx));
        fy.add(mul_rn(fpair, pr.dy));
        fz.add(mul_rn(fpair, pr.dz));
      }
    }
  }
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) {
    fx.shfl_merge(s);
    fy.shfl_merge(s);
    fz.shfl_merge(s);
  }
  double v[1] = {0.0};
  if (active && sub == 0)
    v[0] = residual(fx.value(), fy.value(), fz.value(), target, c, i, fp[i], G, fout);
  write_partials<1>(v, part);
}

// Adjoint, first pass: w_i over atom i's row, the F coefficients' gradient,
// and wf_i = w_i F''_i for the second pass.
template <class Geo, int LPA>
__global__ void __launch_bounds__(kThreads) k_fm_eam_weights(
    Geo g, NbrView nl, int n, const int* __restrict__ types, FitEam e, double rc_sq,
    const double* __restrict__ rho, const double* __restrict__ fpp,
    const double4* __restrict__ G, double* __restrict__ wf) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA, sub = tid % LPA;
  const bool active = i < n;
  const bool multi = e.nt > 1;
  double w = 0.0;
  if (active) {
    const typename Geo::Own o = g.own(i);
    const double4 gi = G[i];
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      const int j = __ldg(nl.nbr + row + k);
      typename Geo::Pair pr;
      g.pair(o, j, pr);
      if (pr.r2 < static_cast<T>(rc_sq)) {
        const double4 gj = ld_d4(G + j);
        T r, rinv;
        double rd;
        g.radius(o, pr, r, rinv, rd);
        double dx;
        const int kk = e.seg(rd, dx);
        const double dr = row_deriv<double>(e.rho_row(multi ? __ldg(types + j) - 1 : 0, kk), dx);
        const double gd = (gi.x - gj.x) * static_cast<double>(pr.dx) +
                          (gi.y - gj.y) * static_cast<double>(pr.dy) +
                          (gi.z - gj.z) * static_cast<double>(pr.dz);
        w -= over_radius(dr * gd, r, rinv);
      }
    }
  }
  w = lane_sum<double, LPA>(w);
  if (active && sub == 0) {
    double dx;
    const int kk = spline_idx(rho[i], e.drho, e.nsf + 1, dx);
    add_deriv_basis(e.gF + 4ll * e.nsf * (multi ? __ldg(types + i) - 1 : 0), e.nsf, kk, dx, w);
    wf[i] = w * fpp[i];
  }
}

// Adjoint, second pass: the phi and rho coefficients, each unordered pair
// once.  The ordered pairs (i, j) and (j, i) meet the same intervals with
// weights that add up: with q = (G_i - G_j) . d / r,
//   phi_p   derivative -q;
//   rho_tj  derivative -q F'_i, value w_i F''_i;
//   rho_ti  derivative -q F'_j, value w_j F''_j
// (one type: one rho spline with both sums), so an unordered pair takes 3 + 4
// scattered adds for one type where the two ordered pairs took 20.  The pass
// is bound by those adds (0.81 cycles per lane and SM in shared memory, 2.1
// in L2).  69 984 atoms, 1.5 M pairs: loss and gradient 280 -> 196 us, of
// which the one-sweep adjoint over ordered pairs took 178.
//
// SHARED (one type): the adds to intervals [k0, k0 + W) go to shared memory,
// one block of 1024 threads per SM over a persistent grid, and out once as a
// block partial ([7][W] doubles, summed by k_fm_eam_window): 148 blocks
// adding their 1 280 x 7 sums to global memory instead took 10 us more.
// Intervals below k0 (pairs closer than k0 * dr) go straight to global
// memory, as every interval does for several types.
constexpr int kPairThreads = 1024;
template <class Geo, int LPA, bool SHARED>
__global__ void __launch_bounds__(SHARED ? kPairThreads : kThreads) k_fm_eam_pairs(
    Geo g, NbrView nl, int n, const int* __restrict__ types, FitEam e, double rc_sq,
    const double4* __restrict__ G, const double* __restrict__ wf, int k0, int W,
    double* __restrict__ part) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  extern __shared__ double sg[];
  if (SHARED) {
    for (int k = threadIdx.x; k < 7 * W; k += blockDim.x) sg[k] = 0.0;
    __syncthreads();
  }
  const int ns = e.nsr;
  const int per_block = blockDim.x / LPA;
  const int sub = threadIdx.x % LPA;
  for (long long ii = static_cast<long long>(blockIdx.x) * per_block + threadIdx.x / LPA; ii < n;
       ii += static_cast<long long>(gridDim.x) * per_block) {
    const int i = static_cast<int>(ii);
    const typename Geo::Own o = g.own(i);
    const double4 gi = G[i];
    const double wi = wf[i];
    const int ti = SHARED ? 0 : __ldg(types + i) - 1;
    const long long row = nl.row(i);
    const int cnt = nl.count(i);
    for (int k = sub; k < cnt; k += LPA) {
      const int j = __ldg(nl.nbr + row + k);
      if (j < i) continue;
      typename Geo::Pair pr;
      g.pair(o, j, pr);
      if (!(pr.r2 < static_cast<T>(rc_sq))) continue;
      const double4 gj = ld_d4(G + j);
      const double wj = __ldg(wf + j);
      T r, rinv;
      double rd;
      g.radius(o, pr, r, rinv, rd);
      double dx;
      const int kk = e.seg(rd, dx);
      const double q = over_radius((gi.x - gj.x) * static_cast<double>(pr.dx) +
                                       (gi.y - gj.y) * static_cast<double>(pr.dy) +
                                       (gi.z - gj.z) * static_cast<double>(pr.dz),
                                   r, rinv);
      if (SHARED && kk >= k0) {
        const double wd = -q * (gi.w + gj.w), wv = wi + wj;
        double* const s = sg + (kk - k0);
        atomicAdd(s, -q);
        atomicAdd(s + W, -2.0 * q * dx);
        atomicAdd(s + 2 * W, -3.0 * q * dx * dx);
        atomicAdd(s + 3 * W, wv);
        atomicAdd(s + 4 * W, fma(wv, dx, wd));
        atomicAdd(s + 5 * W, dx * fma(wv, dx, 2.0 * wd));
        atomicAdd(s + 6 * W, dx * dx * fma(wv, dx, 3.0 * wd));
      } else {
        const int tj = SHARED ? 0 : __ldg(types + j) - 1;
        add_deriv_basis(e.gphi + 4ll * ns * (SHARED ? 0 : pair_index(ti, tj, e.nt)), ns, kk, dx,
                        -q);
        if (ti == tj) {
          add_both_bases(e.grho + 4ll * ns * tj, ns, kk, dx, -q * (gi.w + gj.w), wi + wj);
        } else {
          add_both_bases(e.grho + 4ll * ns * tj, ns, kk, dx, -q * gi.w, wi);
          add_both_bases(e.grho + 4ll * ns * ti, ns, kk, dx, -q * gj.w, wj);
        }
      }
    }
  }
  if (SHARED) {
    __syncthreads();
    double* const o = part + static_cast<long long>(blockIdx.x) * 7 * W;
    for (int k = threadIdx.x; k < 7 * W; k += blockDim.x) o[k] = sg[k];
  }
}

// Adds the block partials of k_fm_eam_pairs to the gradients: 32 columns of
// the 7 W per block, 8 threads sharing a column's nblk records.
__global__ void __launch_bounds__(256) k_fm_eam_window(const double* __restrict__ part, int nblk,
                                                       int W, int k0, int ns,
                                                       double* __restrict__ gphi,
                                                       double* __restrict__ grho) {
  dependent_launch_prologue();
  __shared__ double red[8][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), part_of = threadIdx.x >> 5;
  double v = 0.0;
  if (c < 7 * W) {
#pragma unroll 4
    for (int b = part_of; b < nblk; b += 8) v += part[static_cast<long long>(b) * 7 * W + c];
  }
  red[part_of][threadIdx.x & 31] = v;
  __syncthreads();
  if (part_of == 0 && c < 7 * W) {
    for (int k = 1; k < 8; ++k) v += red[k][threadIdx.x];
    const int coef = c / W, k = k0 + c % W;
    // columns: phi's b, c, d, then rho's a, b, c, d
    double* const g = coef < 3 ? gphi + (coef + 1) * ns + k : grho + (coef - 3) * ns + k;
    *g += v;
  }
}

}  // namespace

// Intervals of the r splines whose gradients a block keeps in shared memory
// (7 doubles each): the top 1280, 70 KiB.
constexpr int kAdjointWindow = 1280;

class Fit {
 public:
  Fit(int nsnap, int natoms, const tdmd_box& box, const double* pos, const int* types,
      double cutoff, int precision);
  ~Fit();
  Fit(const Fit&) = delete;
  Fit& operator=(const Fit&) = delete;
  void set_targets(const double* t);
  void morse(const double* d_prm, double* d_loss, double* d_grad, double* d_forces,
             cudaStream_t s);
  void eam(int ntypes, int nrho, double drho, int nr, double dr, const double* F,
           const double* rho, const double* phi, double* d_loss, double* gF, double* grho,
           double* gphi, double* d_forces, cudaStream_t s);
  long long natoms() const { return m_; }
  int lanes() const { return lpa_; }

 private:
  template <class Fn>
  void with_geo(Fn&& fn) const;
  NbrView view() const { return NbrView{nbr_.data(), nullptr, cnt_.data(), cap_}; }
  // doubles of the adjoint's block partials
  size_t window_size() const {
    return static_cast<size_t>(std::min(sm_count(), ceil_div(m_ * lpa_, kPairThreads))) * 7 *
           kAdjointWindow;
  }

  int nsnap_, n_;
  long long m_;
  bool mixed_;
  double rc_, rc_sq_;
  int lpa_ = 4;
  int cap_ = 0;
  int ncells_ = 0;
  bool has_targets_ = false;
  int max_type_ = 0;
  DevArray<RepDesc> reps_;
  DevArray<RepScale> scales_;
  DevArray<RepImg> imgs_;
  DevArray<int> cell_rep_, rep_;
  DevArray<double4> pos4_;
  DevArray<int4> q_;
  DevArray<int> types_;
  DevArray<int> nbr_, cnt_, status_;
  DevArray<double> target_, rho_, fp_, fpp_, wf_, part_;
  DevArray<double4> G_;      // {dL/dF_i, F'_i}
  DevArray<double4> rec_;    // FP64 {position, F'} gather records
  DevArray<int4> recq_;      // mixed: fixed-point position, F' bits
  DevArray<double4> rows_;   // row copies of the r splines
  DevArray<double> window_;  // block partials of the shared-memory window
  CellListDev cl_;
};

Fit::Fit(int nsnap, int natoms, const tdmd_box& box, const double* pos, const int* types,
         double cutoff, int precision)
    : nsnap_(nsnap), n_(natoms), mixed_(precision == TDMD_MIXED), rc_(cutoff),
      rc_sq_(cutoff * cutoff) {
  TDMD_REQUIRE(nsnap >= 1 && natoms >= 1, "need at least one snapshot and one atom");
  TDMD_REQUIRE(pos && types, "null positions or types");
  TDMD_REQUIRE(cutoff > 0.0, "cutoff must be positive");
  TDMD_REQUIRE(precision == TDMD_FP64 || precision == TDMD_MIXED, "unknown precision");
  m_ = static_cast<long long>(nsnap) * natoms;
  TDMD_REQUIRE(m_ < INT_MAX / 4, "too many atoms");
  const DevBox b = make_devbox(box, cutoff);
  for (int a = 0; a < 3; ++a)
    TDMD_REQUIRE(!b.periodic[a] || b.L[a] > 2.0 * cutoff,
                 "periodic box edge must exceed twice the cutoff");
  for (long long i = 0; i < m_; ++i) {
    TDMD_REQUIRE(types[i] >= 1, "types are 1-based");
    max_type_ = std::max(max_type_, types[i]);
  }
  std::vector<RepDesc> d(static_cast<size_t>(nsnap));
  const int ncell1 = b.nc[0] * b.nc[1] * b.nc[2];
  for (int s = 0; s < nsnap; ++s) {
    RepDesc& r = d[static_cast<size_t>(s)];
    r = RepDesc{};
    r.box = b;
    r.atom0 = s * natoms;
    r.natoms = natoms;
    r.cell0 = s * ncell1;
    r.ncells = ncell1;
    row_filter_band(b, rc_sq_, &r.lo_f, &r.hi_f, &r.wrap);
  }
  ncells_ = nsnap * ncell1;
  const size_t m = static_cast<size_t>(m_);
  std::vector<int> crep(static_cast<size_t>(ncells_)), arep(m);
  for (int s = 0; s < nsnap; ++s) {
    std::fill(crep.begin() + static_cast<long>(s) * ncell1,
              crep.begin() + static_cast<long>(s + 1) * ncell1, s);
    std::fill(arep.begin() + static_cast<long>(s) * natoms,
              arep.begin() + static_cast<long>(s + 1) * natoms, s);
  }
  std::vector<double4> p4(m);
  std::vector<int4> q(m);
  for (size_t i = 0; i < m; ++i) {
    p4[i] = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], static_cast<double>(types[i]));
  }
  const RepScale sc = rep_scale(b);
  const RepImg im = img3(b);
  std::vector<RepScale> scv(static_cast<size_t>(nsnap), sc);
  std::vector<RepImg> imv(static_cast<size_t>(nsnap), im);
  cudaStream_t s = nullptr;
  TDMD_CU(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  try {
    reps_.reserve(d.size());
    scales_.reserve(scv.size());
    imgs_.reserve(imv.size());
    cell_rep_.reserve(crep.size());
    rep_.reserve(m);
    pos4_.reserve(m);
    types_.reserve(m);
    cnt_.reserve(m);
    status_.reserve(4);
    target_.reserve(3 * m);
    G_.reserve(m);
    rho_.reserve(m);
    fp_.reserve(m);
    fpp_.reserve(m);
    wf_.reserve(m);
    if (mixed_)
      recq_.reserve(m);
    else
      rec_.reserve(m);
    TDMD_CU(cudaMemcpyAsync(reps_.data(), d.data(), sizeof(RepDesc) * d.size(),
                            cudaMemcpyHostToDevice, s));
    TDMD_CU(cudaMemcpyAsync(scales_.data(), scv.data(), sizeof(RepScale) * scv.size(),
                            cudaMemcpyHostToDevice, s));
    TDMD_CU(cudaMemcpyAsync(imgs_.data(), imv.data(), sizeof(RepImg) * imv.size(),
                            cudaMemcpyHostToDevice, s));
    TDMD_CU(cudaMemcpyAsync(cell_rep_.data(), crep.data(), sizeof(int) * crep.size(),
                            cudaMemcpyHostToDevice, s));
    TDMD_CU(cudaMemcpyAsync(rep_.data(), arep.data(), sizeof(int) * m, cudaMemcpyHostToDevice, s));
    TDMD_CU(cudaMemcpyAsync(pos4_.data(), p4.data(), sizeof(double4) * m, cudaMemcpyHostToDevice,
                            s));
    TDMD_CU(cudaMemcpyAsync(types_.data(), types, sizeof(int) * m, cudaMemcpyHostToDevice, s));
    if (mixed_) {
      for (size_t i = 0; i < m; ++i) {
        q[i].x = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(
            std::llrint((pos[3 * i] - b.qlo[0]) * b.qinv[0]))));
        q[i].y = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(
            std::llrint((pos[3 * i + 1] - b.qlo[1]) * b.qinv[1]))));
        q[i].z = static_cast<int>(static_cast<uint32_t>(static_cast<unsigned long long>(
            std::llrint((pos[3 * i + 2] - b.qlo[2]) * b.qinv[2]))));
        q[i].w = types[i];
      }
      q_.reserve(m);
      TDMD_CU(cudaMemcpyAsync(q_.data(), q.data(), sizeof(int4) * m, cudaMemcpyHostToDevice, s));
    }
    // Neighbor rows (r_list = cutoff, no skin: positions never move).
    TDMD_CU(cudaMemsetAsync(status_.data(), 0, sizeof(int) * 4, s));
    build_cell_list_batch(cl_, pos4_.data(), rep_.data(), reps_.data(), m_, ncells_, s);
    build_neighbor_rows_batch(cl_, pos4_.data(), reps_.data(), cell_rep_.data(), rc_sq_, nullptr,
                              0, cnt_.data(), status_.data(), s);
    int st[4];
    TDMD_CU(cudaMemcpyAsync(st, status_.data(), sizeof(st), cudaMemcpyDeviceToHost, s));
    TDMD_CU(cudaStreamSynchronize(s));
    cap_ = std::max(8, (st[1] + 7) / 8 * 8);
    nbr_.reserve(static_cast<size_t>(cap_) * m);
    build_neighbor_rows_batch(cl_, pos4_.data(), reps_.data(), cell_rep_.data(), rc_sq_,
                              nbr_.data(), cap_, cnt_.data(), nullptr, s);
    lpa_ = default_lpa(m_);
    // One element may take the shared-memory adjoint: its block partials, at
    // the widest window a call can ask for, so that no call allocates them
    // (0.75 ms of a first gradient).  Morse losses do without, so a device
    // without room for them still gets its handle.
    if (max_type_ == 1) window_.try_reserve(window_size());
    part_.reserve(2 * (static_cast<size_t>(force_blocks(m_, 32)) * kPart + kPart));
    TDMD_CU(cudaStreamSynchronize(s));
  } catch (...) {
    cudaStreamDestroy(s);
    throw;
  }
  cudaStreamDestroy(s);
}

Fit::~Fit() = default;

void Fit::set_targets(const double* t) {
  TDMD_REQUIRE(t, "null targets");
  TDMD_CU(cudaMemcpy(target_.data(), t, sizeof(double) * 3 * static_cast<size_t>(m_),
                     cudaMemcpyHostToDevice));
  has_targets_ = true;
}

template <class Fn>
void Fit::with_geo(Fn&& fn) const {
  if (mixed_)
    fn(GeoQB{q_.data(), rep_.data(), scales_.data()});
  else
    fn(GeoD4B{pos4_.data(), rep_.data(), imgs_.data()});
}

void Fit::morse(const double* d_prm, double* d_loss, double* d_grad, double* d_forces,
                cudaStream_t s) {
  TDMD_REQUIRE(has_targets_, "targets not set");
  TDMD_REQUIRE(d_prm && d_loss, "null parameter or loss pointer");
  const NbrView nl = view();
  const int m = static_cast<int>(m_);
  const int nblk = force_blocks(m_, lpa_);
  const double c = 1.0 / (3.0 * static_cast<double>(m_));
  with_geo([&](auto g) {
    using Geo = decltype(g);
    TDMD_LPA_DISPATCH(lpa_, {
      launch(k_fm_morse_force<Geo, L>, nblk, kThreads, 0, s, g, nl, m, d_prm, rc_sq_,
             target_.data(), c, G_.data(), d_forces, part_.data());
    });
  });
  TDMD_LAUNCH_CHECK();
  double* const part2 = part_.data() + static_cast<size_t>(nblk) * kPart;
  if (d_grad) {
    with_geo([&](auto g) {
      using Geo = decltype(g);
      TDMD_LPA_DISPATCH(lpa_, {
        launch(k_fm_morse_grad<Geo, L>, nblk, kThreads, 0, s, g, nl, m, d_prm, rc_sq_, G_.data(),
               part2);
      });
    });
    TDMD_LAUNCH_CHECK();
  }
  launch(k_fm_sum, d_grad ? 2 : 1, kThreads, 0, s, part_.data(), 1, d_loss, part2, 3, d_grad,
         nblk);
  TDMD_LAUNCH_CHECK();
}

void Fit::eam(int ntypes, int nrho, double drho, int nr, double dr, const double* F,
              const double* rho, const double* phi, double* d_loss, double* gF, double* grho,
              double* gphi, double* d_forces, cudaStream_t s) {
  TDMD_REQUIRE(has_targets_, "targets not set");
  TDMD_REQUIRE(ntypes >= 1 && ntypes <= 64, "ntypes out of range");
  TDMD_REQUIRE(max_type_ <= ntypes, "an atom type exceeds the table's element count");
  // Pairs up to the fit's cutoff evaluate the r tables: past their last knot
  // the cubic of the last interval would be extrapolated.
  TDMD_REQUIRE(rc_ <= static_cast<double>(nr - 1) * dr * (1.0 + 1e-12),
               "the fit's cutoff exceeds the range of the EAM r tables");
  TDMD_REQUIRE(nrho >= 2 && nr >= 2 && drho > 0.0 && dr > 0.0, "bad spline grid");
  TDMD_REQUIRE(F && rho && phi && d_loss, "null coefficient or loss pointer");
  const bool grad = gF || grho || gphi;
  TDMD_REQUIRE(!grad || (gF && grho && gphi), "give all three gradient arrays or none");
  const int npairs = ntypes * (ntypes + 1) / 2;
  const size_t nrows = static_cast<size_t>(ntypes + npairs) * (nr - 1);
  const CallScratch<double4> rows(rows_, nrows, nrows, s);
  // Offsets closer to a knot than the rounding of r / dr (r / dr < nr < 2^31:
  // below 2^-21 dr), or than the cutoff may lie past the last knot, are not
  // decided by the product with 1/dr.
  const double edge = std::max(0x1p-20, 4e-12 * nr);
  const unsigned in_lo = high_word(edge * dr) + 1;
  const unsigned in_hi = high_word((1.0 - edge) * dr);  // offsets below it in the high word
  const FitEam e{F,  rows.data(), gF,       grho,  gphi, ntypes, nrho - 1, nr - 1, drho,
                 dr, 1.0 / dr,    in_lo, in_hi > in_lo ? in_hi - in_lo : 0};
  launch(k_fm_rows, std::min(2 * sm_count(), ceil_div(4ll * (ntypes + npairs) * (nr - 1), 256)),
         256, 0, s, rho, phi, ntypes, npairs, nr - 1, rows.data(), gF,
         4ll * (nrho - 1) * ntypes, grho, gphi);
  TDMD_LAUNCH_CHECK();
  const NbrView nl = view();
  const int m = static_cast<int>(m_);
  const int nblk = force_blocks(m_, lpa_);
  const double c = 1.0 / (3.0 * static_cast<double>(m_));
  // The window of the shared-memory adjoint (one element).
  const int W = std::min(nr - 1, kAdjointWindow);
  const int grid = std::min(sm_count(), ceil_div(m_ * lpa_, kPairThreads));
  std::optional<CallScratch<double>> window;
  if (grad && ntypes == 1)
    window.emplace(window_, window_size(), static_cast<size_t>(grid) * 7 * static_cast<size_t>(W),
                   s);
  auto passes = [&](auto g, auto gf) {
    using Geo = decltype(g);
    using GeoF = decltype(gf);
    TDMD_LPA_DISPATCH(lpa_, {
      launch(k_fm_eam_density<Geo, L>, nblk, kThreads, 0, s, g, nl, m, types_.data(), e, rc_sq_,
             rho_.data(), fp_.data(), fpp_.data(), rec_.data(), recq_.data());
      launch(k_fm_eam_force<GeoF, L>, nblk, kThreads, 0, s, gf, nl, m, types_.data(), e, rc_sq_,
             fp_.data(), target_.data(), c, G_.data(), d_forces, part_.data());
      if (grad) {
        launch(k_fm_eam_weights<Geo, L>, nblk, kThreads, 0, s, g, nl, m, types_.data(), e, rc_sq_,
               rho_.data(), fpp_.data(), G_.data(), wf_.data());
        if (ntypes == 1) {
          const size_t smem = sizeof(double) * 7 * static_cast<size_t>(W);
          auto kern = k_fm_eam_pairs<Geo, L, true>;
          TDMD_CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem)));
          launch(kern, grid, kPairThreads, smem, s, g, nl, m, types_.data(), e, rc_sq_, G_.data(),
                 wf_.data(), (nr - 1) - W, W, window->data());
          launch(k_fm_eam_window, ceil_div(7 * W, 32), 256, 0, s, window->data(), grid, W,
                 (nr - 1) - W, nr - 1, gphi, grho);
        } else {
          launch(k_fm_eam_pairs<Geo, L, false>, nblk, kThreads, 0, s, g, nl, m, types_.data(), e,
                 rc_sq_, G_.data(), wf_.data(), 0, 0, nullptr);
        }
      }
    });
  };
  if (mixed_)
    passes(GeoQB{q_.data(), rep_.data(), scales_.data()},
           GeoQB{recq_.data(), rep_.data(), scales_.data()});
  else
    passes(GeoD4B{pos4_.data(), rep_.data(), imgs_.data()},
           GeoD4BF{rec_.data(), rep_.data(), imgs_.data()});
  TDMD_LAUNCH_CHECK();
  launch(k_fm_sum, 1, kThreads, 0, s, part_.data(), 1, d_loss, nullptr, 0, nullptr, nblk);
  TDMD_LAUNCH_CHECK();
}

}  // namespace tdmd_b200

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace tdmd_b200;

struct tdmd_fit {
  Fit f;
  tdmd_fit(int nsnap, int natoms, const tdmd_box& box, const double* pos, const int* types,
           double cutoff, int precision)
      : f(nsnap, natoms, box, pos, types, cutoff, precision) {}
};

extern "C" {

int32_t tdmd_fit_create(int32_t nsnap, int32_t natoms, const tdmd_box* box,
                        const double* positions, const int32_t* types, double cutoff,
                        int32_t precision, tdmd_fit** out) {
  return guarded([&] {
    TDMD_REQUIRE(out && box, "null argument");
    *out = new tdmd_fit(nsnap, natoms, *box, positions, types, cutoff, precision);
  });
}

int32_t tdmd_fit_destroy(tdmd_fit* f) {
  delete f;
  return TDMD_OK;
}

int32_t tdmd_fit_set_targets(tdmd_fit* f, const double* targets) {
  return guarded([&] {
    TDMD_REQUIRE(f, "null handle");
    f->f.set_targets(targets);
  });
}

int32_t tdmd_fit_morse(tdmd_fit* f, const double* d_params, double* d_loss, double* d_grad,
                       double* d_forces, void* stream) {
  return guarded([&] {
    TDMD_REQUIRE(f, "null handle");
    f->f.morse(d_params, d_loss, d_grad, d_forces, as_stream(stream));
  });
}

int32_t tdmd_fit_eam(tdmd_fit* f, int32_t ntypes, int32_t nrho, double drho, int32_t nr,
                     double dr, const double* d_F, const double* d_rho, const double* d_phi,
                     double* d_loss, double* d_gF, double* d_grho, double* d_gphi,
                     double* d_forces, void* stream) {
  return guarded([&] {
    TDMD_REQUIRE(f, "null handle");
    f->f.eam(ntypes, nrho, drho, nr, dr, d_F, d_rho, d_phi, d_loss, d_gF, d_grho, d_gphi,
             d_forces, as_stream(stream));
  });
}

int32_t tdmd_fit_info(const tdmd_fit* f, int64_t* natoms_total, int32_t* lanes_per_atom) {
  return guarded([&] {
    TDMD_REQUIRE(f, "null handle");
    if (natoms_total) *natoms_total = f->f.natoms();
    if (lanes_per_atom) *lanes_per_atom = f->f.lanes();
  });
}

}  // extern "C"
