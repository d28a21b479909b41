// forces.cuh -- Morse and three-pass EAM force kernels (sm_100a), shared by
// the free-function C ABI (reference array layouts) and the scheduler
// (its own layouts).
//
// Reference kernels (tdmd_Claude): morse_force_kernel
// (src/potentials/device_morse.cu:32-132), eam_density_kernel /
// eam_embedding_kernel / eam_force_kernel (src/potentials/device_eam.cu:
// 72-278), spline_eval / spline_eval_deriv (device_eam.cu:41-66).
//
// Design (B200):
//  * LPA lanes per atom (1..32, a template parameter the autotuner picks):
//    the lanes of a group stride through the atom's neighbor row and merge
//    their partial sums with xor-shuffles; no atomics anywhere.
//  * Geometry policies: FP64 positions (double4 records or the reference's
//    Vec3D AoS, min-image in double), the reference's mixed form (FP64
//    delta cast to FP32), or fixed-point int32 positions whose wrapped
//    difference IS the minimum image (scheduler's mixed path, 16-byte
//    gathers).
//  * Mixed precision: FP32 distances/splines/forces with rsqrt-based 1/r, a
//    refined radius (two floats for the spline offset, FP64 for the Morse
//    exponent), compensated FP32 per-atom sums (Kahan per lane, TwoSum across
//    lanes); energies and virial always accumulate in FP64.
//  * Energy/virial (template EV): per-block FP64 partials reduced later in a
//    fixed order by k_reduce_partials.
//  * EAM splines: the density pass reads rows (a,b,c,d) of rho_t; the force
//    pass reads derivative-ready rows (b, 2c, 3d, a) of every r-spline of one
//    interval side by side (density of each type, then phi of each pair), so
//    a single-type pair's lookups share one 32-byte sector.  The embedding
//    F(rho) is always evaluated in FP64 (one lookup per atom).
//  * Scheduler mixed EAM: the density pass emits a gather record
//    {qx, qy, qz, F'(rho)} per atom; the force pass reads position and F'
//    of a neighbor in one 16-byte load.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "integrate.cuh"
#include "replicas.cuh"

namespace tdmd_b200 {

constexpr int kEvStride = 8;  // doubles per block partial: e, w[6], pad

// --------------------------------------------------------------------------
// Neighbor rows: padded (row = i*cap) or dense CSR (row = row_off[i]).
// --------------------------------------------------------------------------
struct NbrView {
  const int* nbr;
  const int* row_off;  // nullable
  const int* cnt;
  int cap;
  __device__ __forceinline__ long long row(int i) const {
    return row_off ? static_cast<long long>(__ldg(row_off + i)) : static_cast<long long>(i) * cap;
  }
  __device__ __forceinline__ int count(int i) const {
    const int c = __ldg(cnt + i);
    return row_off ? c : (c < cap ? c : cap);
  }
};

// L1 eviction-priority loads: spline rows are re-read by every pair and
// stay resident (evict_last); neighbor indices are read once and bypass L1
// (no_allocate), so they do not push rows and position records out.
__device__ __forceinline__ float4 ld_keep(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::evict_last.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_stream(const int4* p) {
  int4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}

// Neighbors per lane per sweep (U): a lane fetches U indices, then U
// positions, then evaluates U pairs, so its loads overlap.  U is 2 or 4,
// chosen by the autotuner; kU is the choice without tuning.
constexpr int kU = 4;

__device__ __forceinline__ int2 ld_stream2(const int2* p) {
  int2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.s32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "l"(p));
  return v;
}

__device__ __forceinline__ int ld_stream1(const int* p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// The slots of a row that lane sub of an atom's LPA lanes takes in a sweep:
// U consecutive ones in one vector load (kVectorRows), or every LPA-th one,
// so that the lanes of an atom hold consecutive entries.  Consecutive entries
// are mostly neighbors in memory (cell order), so a warp's record gathers
// then touch fewer lines and meet less in a bank (counted on a 131k list, 8
// lanes x 2: 13 lines and 25 bank cycles per 32 FP64 records instead of 17
// and 28), and on dense rows the index loads coalesce.  FP64 and dense rows
// gain (FP64 EAM 131k 5.74 -> 5.64 ms per 50 steps, Morse 256 815 -> 782 us
// per 100, FP64 EAM evaluation of 40k atoms 69.8 -> 65.5 us); the 16-byte
// mixed records do not (131k 3.86 -> 3.92 ms: more index loads than it
// saves), so mixed padded rows keep the vector load, as do 1 to 4 lanes,
// where a lane's own entries fill its sector.  Vector loads need padded rows
// (VEC: 16-byte aligned, capacity a multiple of 4).
template <bool VEC, int LPA, class T>
constexpr bool kVectorRows = VEC && (LPA <= 4 || sizeof(T) == sizeof(float));

// First sweep of lane sub; sweeps advance by U * LPA.
template <bool VEC, int LPA, class T, int U>
__device__ __forceinline__ int first_slot(int sub) {
  return kVectorRows<VEC, LPA, T> ? U * sub : sub;
}

// Indices of the sweep at base < c, -1 past the count.
template <bool VEC, int LPA, class T, int U>
__device__ __forceinline__ void nbr_batch(const NbrView& nl, long long row, int base, int c,
                                          int (&j)[U]) {
  static_assert(U == 2 || U == 4, "neighbor batch: 2 or 4");
  if constexpr (kVectorRows<VEC, LPA, T> && U == 2) {
    const int2 v = ld_stream2(reinterpret_cast<const int2*>(nl.nbr + row + base));
    j[0] = v.x;
    j[1] = base + 1 < c ? v.y : -1;
  } else if constexpr (kVectorRows<VEC, LPA, T>) {
    const int4 v = ld_stream(reinterpret_cast<const int4*>(nl.nbr + row + base));
    j[0] = v.x;
    j[1] = base + 1 < c ? v.y : -1;
    j[2] = base + 2 < c ? v.z : -1;
    j[3] = base + 3 < c ? v.w : -1;
  } else {
    const int* const r = nl.nbr + row + base;
#pragma unroll
    for (int u = 0; u < U; ++u)
      j[u] = base + u * LPA < c ? (VEC ? ld_stream1(r + u * LPA) : __ldg(r + u * LPA)) : -1;
  }
}

// --------------------------------------------------------------------------
// Geometry policies.  own(i) loads atom i once; pair(own, j, p) fills p with
// r_i - r_j after the minimum image and r^2 in the policy's arithmetic type
// T; radius(own, p, r, rinv, rd) gives |r_i - r_j| and its inverse as T and as
// an FP64 value rd that the Morse exponent and the fits use, radius2 the same
// refined radius as r + corr in T for the spline offset.  In
// FP32, r itself carries an absolute error of ~ulp(r) = 2.4e-7 A at
// r ~ 2.5 A, which moves the spline argument and, through the large pair
// forces that cancel in each atom's net force, dominates the mixed-precision
// force error; rd removes that term (one Newton step in FP64 from the FP32
// root, with the residual r^2 - r_f^2 taken from FP64 r^2).
// --------------------------------------------------------------------------
struct PairD {
  double dx, dy, dz, r2;
};

// FP64 minimum image of the pair deltas: h is L/2 on a periodic axis and
// +infinity on a free one, so one compare of |d| and one add of -+L give the
// bits of min_image1's two compares (9 FP64 operations a pair instead of 15).
struct Img3 {
  double L[3], h[3];
};
__host__ inline Img3 img3(const DevBox& b) {
  Img3 m{};
  for (int a = 0; a < 3; ++a) {
    m.L[a] = b.L[a];
    m.h[a] = b.periodic[a] ? b.halfL[a] : HUGE_VAL;
  }
  return m;
}
__device__ __forceinline__ double image1(double d, double L, double h) {
  return fabs(d) > h ? d - copysign(L, d) : d;
}

// r = sqrt(x) and rinv = 1/sqrt(x) in FP64 from the FP32 reciprocal root y of
// x by one third-order Householder step: with g = x y, h = y/2 and
// e = 1/2 - g h (one rounding: FMA), g and h are multiplied by
// (1 - 2e)^(-1/2) = 1 + e + 3/2 e^2 + O(e^3).  |e| < 1e-6 (2^-22.9 of the
// seed, the rounding of x), so the truncation is below 2^-58; then one Newton
// correction of the root with its exact residual x - r^2 (FMA) rounds it as
// sqrt does, and div_r the quotient as a division does.  15 FP64 operations
// without a branch for a force pair, where sqrt(x) and two divisions by r
// (spline interval, force) took about 40 with a branch each: Morse 256 atoms
// FP64 847 -> 814 us per 100 steps, EAM 131k FP64 6.58 -> 6.47 ms per 50, one
// EAM evaluation of 40k atoms 76 -> 72 us; same error against 64 bits.
// Outside [2^-100, 2^100) (the seed's range; no listed pair of a physical
// system) the library root is taken.
__device__ __forceinline__ void radius_d(double x, double& r, double& rinv) {
  const unsigned hi = static_cast<unsigned>(__double2hiint(x));
  if (hi - 0x39b00000u < 0x46300000u - 0x39b00000u) {
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(static_cast<float>(x)));
    const double y = static_cast<double>(y0);
    const double g = x * y, h = 0.5 * y;
    const double e = fma(-g, h, 0.5);
    const double t = e * fma(1.5, e, 1.0);
    const double r0 = fma(g, t, g), h1 = fma(h, t, h);
    r = fma(fma(-r0, r0, x), h1, r0);
    rinv = h1 + h1;
  } else {
    r = sqrt(x);
    rinv = 1.0 / r;
  }
}

// |r_i - r_j| alone.
__device__ __forceinline__ double root_d(double x) {
  double r, rinv;
  radius_d(x, r, rinv);
  return r;
}

// x / r: FP64 corrects the product with 1/r by its exact remainder (the
// division's rounding; an infinite quotient has no remainder and stays, as the
// division leaves it -- a predicate on the correction, which costs nothing
// measurable, where selecting between the two took 0.5 % of the FP64 passes);
// FP32 multiplies by rsqrt.
__device__ __forceinline__ double div_r(double x, double r, double rinv) {
  double q = x * rinv;
  const double rem = fma(-q, r, x);
  asm("{\n .reg .pred finite;\n .reg .b32 lo, hi;\n"
      " mov.b64 {lo, hi}, %0;\n and.b32 hi, hi, 0x7ff00000;\n"
      " setp.ne.u32 finite, hi, 0x7ff00000;\n"
      " @finite fma.rn.f64 %0, %1, %2, %0;\n}"
      : "+d"(q)
      : "d"(rem), "d"(rinv));
  return q;
}
__device__ __forceinline__ float div_r(float x, float /*r*/, float rinv) { return x * rinv; }

struct PairF {
  float dx, dy, dz, r2;
  double r2d;  // FP64 r^2
};

// res: the FP64 r^2 of the exact fixed-point delta minus r2, rounded to
// float -- all that the radius refinement needs of the delta, so a pair in
// flight holds six words instead of eight.
struct PairQ {
  float dx, dy, dz, r2;
  float res;
  int w;  // the neighbor's 4th word
};

// 1/sqrt of a fixed-point pair's r^2: zero or at least (L/2^32)^2, so the
// reciprocal root needs none of rsqrtf's rescaling of subnormals (two
// predicated multiplications and a compare a pair; same bits).
__device__ __forceinline__ float rsqrt_q(float r2) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
  return y;
}

// FP64 residual (exact r^2 of the fixed-point deltas) - r2.  When the
// three axes share one step (iso), the squares are summed exactly in 64-bit
// integers (|d| <= 2^31: each square <= 2^62, the sum < 2^64) and scaled
// once; otherwise each axis is scaled in FP64.
__device__ __forceinline__ float q_residual(int ix, int iy, int iz, int iso, double s2x,
                                            double s2y, double s2z, float r2) {
  if (iso) {
    const unsigned long long q2 = static_cast<unsigned long long>(static_cast<long long>(ix) * ix) +
                                  static_cast<unsigned long long>(static_cast<long long>(iy) * iy) +
                                  static_cast<unsigned long long>(static_cast<long long>(iz) * iz);
    return static_cast<float>(fma(__ull2double_rn(q2), s2x, -static_cast<double>(r2)));
  }
  const double x = ix, y = iy, z = iz;
  return static_cast<float>(x * x * s2x + y * y * s2y + z * z * s2z - static_cast<double>(r2));
}

// |r| and 1/|r| in FP32 and the FP64-refined radius from a PairQ: with
// r = sqrt(r2) in FP32, r2d - r*r = res + (r2 - r*r), the second term exact
// by FMA; one Newton step rd = r + (r2d - r*r) / (2r).
__device__ __forceinline__ void radius_q(float r2, float res, float& r, float& rinv, double& rd) {
  rinv = rsqrt_q(r2);
  r = r2 * rinv;
  const float corr = (res + fmaf(-r, r, r2)) * 0.5f * rinv;
  rd = static_cast<double>(r) + static_cast<double>(corr);
}

// The same refined radius as a pair of floats r + corr.
__device__ __forceinline__ void radius_q2(float r2, float res, float& r, float& rinv,
                                          float& corr) {
  rinv = rsqrt_q(r2);
  r = r2 * rinv;
  corr = (res + fmaf(-r, r, r2)) * 0.5f * rinv;
}
__device__ __forceinline__ void radius_f2(float r2, double r2d, float& r, float& rinv,
                                          float& corr) {
  rinv = rsqrtf(r2);
  r = r2 * rinv;
  corr = static_cast<float>(fma(-static_cast<double>(r), r, r2d)) * 0.5f * rinv;
}

__device__ __forceinline__ void radius_f(float r2, double r2d, float& r, float& rinv, double& rd) {
  rinv = rsqrtf(r2);
  r = r2 * rinv;
  rd = static_cast<double>(r) +
       static_cast<double>(static_cast<float>(fma(-static_cast<double>(r), r, r2d)) * 0.5f * rinv);
}

// Geometries whose density pass may write FP64 gather records {x, y, z, F'}
// (their own atom's position as x, y, z members) declare kD4Out.
template <class G, class = void>
struct has_d4out : std::false_type {};
template <class G>
struct has_d4out<G, std::void_t<decltype(G::kD4Out)>> : std::bool_constant<G::kD4Out> {};

struct GeoD4 {  // FP64, scheduler layout double4 {x,y,z,type}
  using T = double;
  static constexpr bool kD4Out = true;
  static constexpr bool kRecords = false;  // no fixed-point gather records
  using Own = double3;
  using Pair = PairD;
  const double4* p;
  Img3 m;
  __device__ __forceinline__ double3 load(int i) const {
    const double4 a = ld_d4(p + i);
    return make_double3(a.x, a.y, a.z);
  }
  __device__ __forceinline__ Own own(int i) const { return load(i); }
  __device__ __forceinline__ void pair(const Own& o, int j, Pair& pr) const {
    const double3 q = load(j);
    pr.dx = image1(o.x - q.x, m.L[0], m.h[0]);
    pr.dy = image1(o.y - q.y, m.L[1], m.h[1]);
    pr.dz = image1(o.z - q.z, m.L[2], m.h[2]);
    pr.r2 = pr.dx * pr.dx + pr.dy * pr.dy + pr.dz * pr.dz;
  }
  __device__ __forceinline__ void radius(const Own&, const Pair& pr, T& r, T& rinv,
                                         double& rd) const {
    radius_d(pr.r2, r, rinv);
    rd = r;
  }
  __device__ __forceinline__ void radius2(const Own&, const Pair& pr, T& r, T& rinv,
                                          T& corr) const {
    radius_d(pr.r2, r, rinv);
    corr = 0.0;
  }
  __device__ __forceinline__ T radius_fast(const Pair& pr) const { return root_d(pr.r2); }
};

// FP64 pair from a gather record: the neighbor's F'(rho) rides along.
struct PairDF {
  double dx, dy, dz, r2;
  double fw;
};

// FP64, scheduler gather records double4 {x, y, z, F'(rho)} written by the
// density pass: the force pass reads a neighbor's position and F' with one
// 32-byte load instead of a position record plus a separate F' gather.
struct GeoD4F {
  using T = double;
  static constexpr bool kRecords = false;
  using Own = double3;
  using Pair = PairDF;
  const double4* p;
  Img3 m;
  __device__ __forceinline__ Own own(int i) const {
    const double4 a = ld_d4(p + i);
    return make_double3(a.x, a.y, a.z);
  }
  __device__ __forceinline__ void pair(const Own& o, int j, Pair& pr) const {
    const double4 q = ld_d4(p + j);
    pr.dx = image1(o.x - q.x, m.L[0], m.h[0]);
    pr.dy = image1(o.y - q.y, m.L[1], m.h[1]);
    pr.dz = image1(o.z - q.z, m.L[2], m.h[2]);
    pr.r2 = pr.dx * pr.dx + pr.dy * pr.dy + pr.dz * pr.dz;
    pr.fw = q.w;
  }
  __device__ __forceinline__ void radius2(const Own&, const Pair& pr, T& r, T& rinv,
                                          T& corr) const {
    radius_d(pr.r2, r, rinv);
    corr = 0.0;
  }
  // F'(rho_j) of a pair's record
  __device__ __forceinline__ double gather_fp(const Pair& pr, int /*tmask*/) const {
    return pr.fw;
  }
};

struct GeoAoS64 {  // FP64, reference Vec3D AoS
  using T = double;
  static constexpr bool kD4Out = true;
  static constexpr bool kRecords = false;
  using Own = double3;
  using Pair = PairD;
  const double* p;
  Img3 m;
  __device__ __forceinline__ double3 load(int i) const {
    const double* q = p + 3ll * i;
    return make_double3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
  }
  __device__ __forceinline__ Own own(int i) const { return load(i); }
  __device__ __forceinline__ void pair(const Own& o, int j, Pair& pr) const {
    const double3 q = load(j);
    pr.dx = image1(o.x - q.x, m.L[0], m.h[0]);
    pr.dy = image1(o.y - q.y, m.L[1], m.h[1]);
    pr.dz = image1(o.z - q.z, m.L[2], m.h[2]);
    pr.r2 = pr.dx * pr.dx + pr.dy * pr.dy + pr.dz * pr.dz;
  }
  __device__ __forceinline__ void radius(const Own&, const Pair& pr, T& r, T& rinv,
                                         double& rd) const {
    radius_d(pr.r2, r, rinv);
    rd = r;
  }
  __device__ __forceinline__ void radius2(const Own&, const Pair& pr, T& r, T& rinv,
                                          T& corr) const {
    radius_d(pr.r2, r, rinv);
    corr = 0.0;
  }
  __device__ __forceinline__ T radius_fast(const Pair& pr) const { return root_d(pr.r2); }
};

// Mixed on the reference layout (free functions): the delta is formed in
// FP64 and min-imaged there, then cast to FP32 (the reference's
// relative-coordinate form, device_morse.cu:58-73, without its FP32
// min-image step).
struct GeoAoS32 {
  using T = float;
  static constexpr bool kRecords = false;
  using Own = double3;
  using Pair = PairF;
  const double* p;
  Img3 m;
  __device__ __forceinline__ double3 load(int i) const {
    const double* q = p + 3ll * i;
    return make_double3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
  }
  __device__ __forceinline__ Own own(int i) const { return load(i); }
  __device__ __forceinline__ void pair(const Own& o, int j, Pair& pr) const {
    const double3 q = load(j);
    const double x = image1(o.x - q.x, m.L[0], m.h[0]);
    const double y = image1(o.y - q.y, m.L[1], m.h[1]);
    const double z = image1(o.z - q.z, m.L[2], m.h[2]);
    pr.dx = static_cast<float>(x);
    pr.dy = static_cast<float>(y);
    pr.dz = static_cast<float>(z);
    pr.r2d = x * x + y * y + z * z;
    pr.r2 = static_cast<float>(pr.r2d);
  }
  __device__ __forceinline__ void radius(const Own&, const Pair& pr, T& r, T& rinv,
                                         double& rd) const {
    radius_f(pr.r2, pr.r2d, r, rinv, rd);
  }
  __device__ __forceinline__ void radius2(const Own&, const Pair& pr, T& r, T& rinv,
                                          T& corr) const {
    radius_f2(pr.r2, pr.r2d, r, rinv, corr);
  }
  __device__ __forceinline__ T radius_fast(const Pair& pr) const { return pr.r2 * rsqrtf(pr.r2); }
};

// Mixed, scheduler layout: fixed-point int4 records {qx,qy,qz,w}.  The
// wrapped int32 difference is the exact minimum-image delta in units of
// Lq/2^32; FP32 components come from one conversion each, the FP64 r^2 from
// the exact integers (only for pairs inside the cutoff).  w is the type
// (position records) or F'(rho) bits (the EAM force-pass gather records).
struct GeoQ {
  using T = float;
  using Own = int4;
  using Pair = PairQ;
  static constexpr bool kRecords = true;  // own() is the atom's fixed-point record
  const int4* q;
  float s[3];
  double s2[3];  // (Lq/2^32)^2 per axis
  int iso;       // one step on all three axes
  __device__ __forceinline__ Own own(int i) const { return __ldg(q + i); }
  __device__ __forceinline__ int4 record(const Own& o) const { return o; }
  __device__ __forceinline__ void pair(const Own& o, int j, Pair& pr) const {
    const int4 b = __ldg(q + j);
    const int ix = o.x - b.x, iy = o.y - b.y, iz = o.z - b.z;
    pr.w = b.w;
    pr.dx = __fmul_rn(__int2float_rn(ix), s[0]);
    pr.dy = __fmul_rn(__int2float_rn(iy), s[1]);
    pr.dz = __fmul_rn(__int2float_rn(iz), s[2]);
    pr.r2 = pr.dx * pr.dx + pr.dy * pr.dy + pr.dz * pr.dz;
    pr.res = q_residual(ix, iy, iz, iso, s2[0], s2[1], s2[2], pr.r2);
  }
  __device__ __forceinline__ void radius(const Own&, const Pair& pr, T& r, T& rinv,
                                         double& rd) const {
    radius_q(pr.r2, pr.res, r, rinv, rd);
  }
  __device__ __forceinline__ void radius2(const Own&, const Pair& pr, T& r, T& rinv,
                                          T& corr) const {
    radius_q2(pr.r2, pr.res, r, rinv, corr);
  }
  __device__ __forceinline__ T radius_fast(const Pair& pr) const { return pr.r2 * rsqrt_q(pr.r2); }
  // F'(rho_j) of a gather record: the 4th word's float bits, type bits cleared
  __device__ __forceinline__ float gather_fp(const Pair& pr, int tmask) const {
    return __int_as_float(pr.w & ~tmask);
  }
};

__host__ inline GeoQ make_geoq(const int4* q, const DevBox& b) {
  return GeoQ{q,
              {b.qscale[0], b.qscale[1], b.qscale[2]},
              {b.qstep[0] * b.qstep[0], b.qstep[1] * b.qstep[1], b.qstep[2] * b.qstep[2]},
              b.qstep[0] == b.qstep[1] && b.qstep[1] == b.qstep[2]};
}

__host__ inline GeoAoS32 make_geo_aos32(const double* p, const DevBox& b) {
  return GeoAoS32{p, img3(b)};
}

// --------------------------------------------------------------------------
// Accumulators: plain double (FP64) or compensated float (mixed: Kahan per
// lane -- 4 flops per term, error bounded by 2 eps sum|x| whatever the
// number of terms -- and error-free TwoSum when lanes merge).
// --------------------------------------------------------------------------
template <class T>
struct Acc;
template <>
struct Acc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ void shfl_merge(int o) { s += __shfl_xor_sync(0xffffffffu, s, o); }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<float> {
  float s = 0.f, c = 0.f;  // running sum, compensation (subtracted)
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
  __device__ __forceinline__ void shfl_merge(int o) {
    const float os = __shfl_xor_sync(0xffffffffu, s, o);
    const float oc = __shfl_xor_sync(0xffffffffu, c, o);
    // (s - c) + (os - oc) with TwoSum on the leading parts.
    const float t = __fadd_rn(s, os);
    const float z = __fsub_rn(t, s);
    const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(os, z));
    s = t;
    c = __fsub_rn(__fadd_rn(c, oc), e);
  }
  __device__ __forceinline__ double value() const {
    return static_cast<double>(s) - static_cast<double>(c);
  }
};

__device__ __forceinline__ double mul_rn(double a, double b) { return a * b; }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// Force output: AoS float3 or double3.
template <class F>
struct ForceOut {
  F* f;
  __device__ __forceinline__ void store(int i, double x, double y, double z) const {
    f[3ll * i] = static_cast<F>(x);
    f[3ll * i + 1] = static_cast<F>(y);
    f[3ll * i + 2] = static_cast<F>(z);
  }
};

// Accumulating force output (the per-zone form: a zone's forces are added to
// what the caller zeroed, compute_morse_gpu_zone, device_morse_zone.cu).
template <class F>
struct ForceAdd {
  F* f;
  __device__ __forceinline__ void store(int i, double x, double y, double z) const {
    f[3ll * i] += static_cast<F>(x);
    f[3ll * i + 1] += static_cast<F>(y);
    f[3ll * i + 2] += static_cast<F>(z);
  }
};

// A geometry whose own atoms start at `first` of the position array; the
// neighbors j of a row stay global indices.  A kernel over atoms
// [first, first + n) then reads its rows, counts and outputs through views
// shifted by first.
template <class G>
struct GeoShift : G {
  int first;
  __device__ __forceinline__ typename G::Own own(int i) const { return G::own(first + i); }
};

// Per-block FP64 energy/virial partials (thread 0 writes 8 doubles).
__device__ __forceinline__ void write_ev_partials(double e, const double (&w)[6],
                                                  double* __restrict__ partials) {
  __shared__ double red[32 * 7];
  double v[7] = {e, w[0], w[1], w[2], w[3], w[4], w[5]};
  block_sum<7>(v, red);
  if (threadIdx.x == 0) {
    double* o = partials + static_cast<long long>(blockIdx.x) * kEvStride;
#pragma unroll
    for (int k = 0; k < 7; ++k) o[k] = v[k];
    o[7] = 0.0;
  }
}

template <class T>
__device__ __forceinline__ void add_virial(double (&w)[6], T fpair, T dx, T dy, T dz) {
  const double hf = 0.5 * static_cast<double>(fpair);
  const double ddx = dx, ddy = dy, ddz = dz;
  w[0] += hf * ddx * ddx;
  w[1] += hf * ddy * ddy;
  w[2] += hf * ddz * ddz;
  w[3] += hf * ddx * ddy;
  w[4] += hf * ddx * ddz;
  w[5] += hf * ddy * ddz;
}

// The next step's fused kick + drift, applied by a force pass to each atom
// right after its force: v += dt F/(m mvv2e), x += dt v with the
// single-image wrap, fixed-point record refreshed (fused_kick_drift_kernel,
// device_velocity_verlet.cu:88-130, full kick).  The EAM force passes read
// gather records, never the positions they update; Morse reads the positions
// themselves, so it writes the new ones to a second buffer (ALT).
struct KickDrift {
  double4* pos4;
  int4* q;
  double* v;
  const int* types;
  const double* inv_mm;  // 1 / (m mvv2e) per type
  double dt;
  long long* step;       // device step counter, +1 per kick-drift (nullable)
  DevBox b;
  // Batched replicas: atom i's box is reps[rep[i]].box instead of b.
  const int* rep;
  const RepDesc* reps;
  // ALT: where the new positions and fixed-point records go.
  double4* pos4_alt = nullptr;
  int4* q_alt = nullptr;
};

// FT: the force type (float: mixed, also refreshes the fixed-point record;
// double: FP64, which keeps no fixed-point copy).
template <bool ALT, class FT>
__device__ __forceinline__ void kick_drift_atom(const KickDrift& k, int i, FT fx, FT fy, FT fz) {
  const DevBox& b = k.reps ? k.reps[__ldg(k.rep + i)].box : k.b;
  const int t = __ldg(k.types + i);
  const double factor = k.dt * __ldg(k.inv_mm + t);
  double vx = k.v[3ll * i], vy = k.v[3ll * i + 1], vz = k.v[3ll * i + 2];
  vx += factor * static_cast<double>(fx);
  vy += factor * static_cast<double>(fy);
  vz += factor * static_cast<double>(fz);
  double4 p = k.pos4[i];
  p.x = wrap_single(p.x + k.dt * vx, b.lo[0], b.L[0], b.periodic[0]);
  p.y = wrap_single(p.y + k.dt * vy, b.lo[1], b.L[1], b.periodic[1]);
  p.z = wrap_single(p.z + k.dt * vz, b.lo[2], b.L[2], b.periodic[2]);
  k.v[3ll * i] = vx;
  k.v[3ll * i + 1] = vy;
  k.v[3ll * i + 2] = vz;
  (ALT ? k.pos4_alt : k.pos4)[i] = p;
  if constexpr (sizeof(FT) == sizeof(float))
    (ALT ? k.q_alt : k.q)[i] =
        make_int4(encode_q(p.x, b.qlo[0], b.qinv[0]), encode_q(p.y, b.qlo[1], b.qinv[1]),
                  encode_q(p.z, b.qlo[2], b.qinv[2]), t);
}

// --------------------------------------------------------------------------
// Morse, MorsePair::compute (src/potentials/morse.hpp:37-55) on the full
// list: F_i = sum_j fpair(r_ij) (r_i - r_j), energy 1/2 U per listed pair.
// --------------------------------------------------------------------------
template <class T>
struct MorseP {
  T d, alpha, r0, rc_sq;
  double r0d;
};

// EV: 0 forces only; 1 also energy + virial into per-block partials and,
// where pe_atom is given, per-atom energies; 2 forces + per-atom energies.
// KD: then the next step's kick + drift of the same atom, the new positions
// into the second buffers: one launch and one pass over the forces less per
// step (256 atoms FP64: 672 -> 612 us per 100 steps; 64 replicas, 142k atoms,
// mixed: 1 %).
template <class Geo, int LPA, int U, int EV, bool VEC, class F, class Out = ForceOut<F>,
          bool KD = false>
__global__ void __launch_bounds__(256) k_morse(Geo g, NbrView nl, int n,
                                               MorseP<typename Geo::T> mp, Out out,
                                               double* __restrict__ partials,
                                               double* __restrict__ pe_atom, KickDrift kd = {}) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA;
  const int sub = tid % LPA;
  const bool active = i < n;
  Acc<T> fx, fy, fz;
  double pe = 0.0;
  double w[6] = {0, 0, 0, 0, 0, 0};
  if (active) {
    const typename Geo::Own o = g.own(i);
    const long long row = nl.row(i);
    const int c = nl.count(i);
    const T two_d_alpha = T(2) * mp.d * mp.alpha;
    for (int base = first_slot<VEC, LPA, T, U>(sub); base < c; base += U * LPA) {
      int jj[U];
      nbr_batch<VEC, LPA, T>(nl, row, base, c, jj);
      typename Geo::Pair pr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (jj[u] >= 0)
          g.pair(o, jj[u], pr[u]);
        else
          pr[u].r2 = mp.rc_sq;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (pr[u].r2 < mp.rc_sq) {
          T r, rinv;
          double rd;
          g.radius(o, pr[u], r, rinv, rd);
          const T ex = exp(-mp.alpha * static_cast<T>(rd - mp.r0d));
          const T ome = T(1) - ex;
          const T fpair = -div_r(two_d_alpha * ome * ex, r, rinv);
          fx.add(mul_rn(fpair, pr[u].dx));
          fy.add(mul_rn(fpair, pr[u].dy));
          fz.add(mul_rn(fpair, pr[u].dz));
          if (EV) {
            pe += 0.5 * static_cast<double>(mp.d * (ome * ome - T(1)));
            if (EV == 1) add_virial(w, fpair, pr[u].dx, pr[u].dy, pr[u].dz);
          }
        }
      }
    }
  }
#pragma unroll
  for (int o = LPA / 2; o > 0; o >>= 1) {
    fx.shfl_merge(o);
    fy.shfl_merge(o);
    fz.shfl_merge(o);
  }
  if (active && sub == 0) {
    out.store(i, fx.value(), fy.value(), fz.value());
    if constexpr (KD)
      kick_drift_atom<true>(kd, i, static_cast<F>(fx.value()), static_cast<F>(fy.value()),
                            static_cast<F>(fz.value()));
  }
  if (KD && kd.step && blockIdx.x == 0 && threadIdx.x == 0) *kd.step += 1;
  if (EV) {
    // per-atom energy (nullable): the lanes' sums merged pairwise
    if (pe_atom) {
      double pa = pe;
#pragma unroll
      for (int o = LPA / 2; o > 0; o >>= 1) pa += __shfl_xor_sync(0xffffffffu, pa, o);
      if (active && sub == 0) pe_atom[i] = pa;
    }
    if (EV == 1 && partials) write_ev_partials(pe, w, partials);
  }
}

// --------------------------------------------------------------------------
// EAM tables on the device.
// --------------------------------------------------------------------------
template <class T>
struct V4;
template <>
struct V4<double> {
  using type = double4;
};
template <>
struct V4<float> {
  using type = float4;
};

template <class T>
struct EamDev {
  const typename V4<T>::type* dtab;  // [(nr-1) * nt] (a, b, c, d) of rho_t
  const typename V4<T>::type* rtab;  // [(nr-1) * S]  (b, 2c, 3d, a), S = nt + npairs
  const double4* ftab;               // [nt * (nrho-1)] (a, b, c, d) of F_t, FP64
  int ntypes, S, nr, nrho;
  T dr, inv_dr, rc_sq;
  double drho;
  // FP32 path: the FP64 knot spacing less dr (its rounding), so that the
  // spline offset r - idx*dr carries no error proportional to idx (the
  // same sign for every pair of a neighbor shell, which summed into a
  // bias of the embedding energy).
  T dr_lo;
  // Multi-type mixed path: the low tbits mantissa bits of the gather
  // record's F'(rho) word hold the atom's 0-based type (a relative change of
  // F' below 2^(tbits-23)), so the force pass gathers no type; 0 = types are
  // gathered (one type, or more than 16).
  int tbits;
  // One type, FP64: the six derivative coefficients of a bin as
  // (rho' b, 2c, 3d, phi' b) and (phi' 2c, 3d), and phi's a for the energy.
  const double4* d4 = nullptr;
  const double2* d2 = nullptr;
  const double* da = nullptr;
  int wide = 0;  // read by the launches: the table takes the WIDE kernels (spline_at)
};

__device__ __forceinline__ int phi_slot(int ti, int tj, int nt) {
  if (ti > tj) {
    const int t = ti;
    ti = tj;
    tj = t;
  }
  return nt + ti * nt - ti * (ti + 1) / 2 + tj;
}

// Interval index and offset, SplineTable::eval (eam_alloy.cpp:52-61):
// idx = int((r - rmin)/dr) clamped to [0, n-2], dx = r - idx*dr (rmin = 0).
__device__ __forceinline__ int spline_idx(double r, double dr, int n, double& dx) {
  int idx = static_cast<int>(r / dr);
  idx = idx < 0 ? 0 : (idx > n - 2 ? n - 2 : idx);
  dx = r - static_cast<double>(idx) * dr;
  return idx;
}

// The same interval from r * (1/dr) without the division: floor(q) as the
// round-to-nearest of q - 1/2 in the low word of q - 1/2 + 1.5 * 2^52, whose
// difference from 1.5 * 2^52 is the interval as a double (no conversions).
// Where q is within a rounding of a knot the neighboring interval may be
// taken (every other exact knot goes to the one below): only for splines whose
// value and derivative are continuous, as build_spline's are, so that the
// result changes by a rounding only.  0 <= q < 2^31.
__device__ __forceinline__ int spline_idx_mul(double r, double dr, double inv_dr, int n,
                                              double& dx) {
  constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
  const double z = fma(r, inv_dr, -0.5) + kRound;
  int idx = __double2loint(z);
  dx = fma(-(z - kRound), dr, r);
  if (static_cast<unsigned>(idx) > static_cast<unsigned>(n - 2)) {
    idx = idx < 0 ? 0 : n - 2;
    dx = r - static_cast<double>(idx) * dr;
  }
  return idx;
}

// Interval of r in FP32 and the same number as a float, as spline_idx_mul has
// it in FP64: no conversions, which run at a quarter of the rate of the
// additions that replace them.  0 <= r / dr < 2^22, and beyond the table.
__device__ __forceinline__ int spline_interval(float r, const EamDev<float>& e, float& fi) {
  constexpr float kRound = 12582912.f;  // 1.5 * 2^23
  const float z = __fadd_rn(fmaf(r, e.inv_dr, -0.5f), kRound);
  int idx = __float_as_int(z) - 0x4B400000;
  fi = __fsub_rn(z, kRound);
  if (static_cast<unsigned>(idx) > static_cast<unsigned>(e.nr - 2)) {
    idx = idx < 0 ? 0 : e.nr - 2;
    fi = static_cast<float>(idx);
  }
  return idx;
}

// Interval from r, offset from the refined radius r + corr (FP32: the knot
// spacing as dr + dr_lo, so that the offset rounds at its own size, below
// 2e-10 A; force, energy and density errors against FP64 are those of an FP64
// offset to four digits, 500 to 10 000 knots).  Without the FP64 radius, whose
// four conversions and two FP64 operations a pair sat in the chain from
// distance to spline row, and with the intervals above: mixed EAM 131k 3.87 ->
// 3.82 ms per 50 steps, 1.05 M atoms 11.89 -> 11.73 ms per 20; ternary 55k NVT
// and 2 767 atoms within their spread.
//
// WIDE: tables beyond the range of these intervals -- 2^22 knots and more in
// FP32, a cutoff 2^31 spacings and more away in FP64 -- find them by division
// and conversion, the offset in FP64.  Kernels of their own (EamDev::wide, by the
// launch): the same cases on a rare branch here cost every mixed pass
// 0.3-0.5 % and the multi-type force pass 1.6 %, and moved what the autotuner
// picks for 4 M ternary atoms (24.5 -> 26.0 ms a window).
template <bool WIDE>
__device__ __forceinline__ int spline_at(double r, double /*corr*/, const EamDev<double>& e,
                                         double& sx) {
  if constexpr (WIDE) return spline_idx(r, e.dr, e.nr, sx);
  return spline_idx_mul(r, e.dr, e.inv_dr, e.nr, sx);
}
template <bool WIDE>
__device__ __forceinline__ int spline_at(float r, float corr, const EamDev<float>& e, float& sx) {
  if constexpr (WIDE) {
    const int idx = min(static_cast<int>(r * e.inv_dr), e.nr - 2);
    sx = static_cast<float>(fma(-static_cast<double>(idx),
                                static_cast<double>(e.dr) + static_cast<double>(e.dr_lo),
                                static_cast<double>(r) + static_cast<double>(corr)));
    return idx;
  }
  float fi;
  const int idx = spline_interval(r, e, fi);
  sx = __fadd_rn(fmaf(-fi, e.dr, r), fmaf(-fi, e.dr_lo, corr));
  return idx;
}

// Interval and offset from r alone (density pass).
template <bool WIDE, class T>
__device__ __forceinline__ int spline_fast(double r, const EamDev<T>& e, double& sx) {
  return spline_at<WIDE>(r, 0.0, e, sx);
}
template <bool WIDE, class T>
__device__ __forceinline__ int spline_fast(float r, const EamDev<T>& e, float& sx) {
  if constexpr (WIDE) return spline_at<true>(r, 0.f, e, sx);
  float fi;
  const int idx = spline_interval(r, e, fi);
  sx = fmaf(-fi, e.dr_lo, fmaf(-fi, e.dr, r));
  return idx;
}

// (a, b, c, d) rows: value a + x(b + x(c + x d)), derivative b + x(2c + 3d x).
template <class C, class T>
__device__ __forceinline__ T spl_val(const C& c, T dx) {
  return c.x + dx * (c.y + dx * (c.z + dx * c.w));
}
template <class C, class T>
__device__ __forceinline__ T spl_der(const C& c, T dx) {
  return c.y + dx * (T(2) * c.z + dx * T(3) * c.w);
}
// (b, 2c, 3d, a) rows.
template <class C, class T>
__device__ __forceinline__ T dspl_der(const C& c, T dx) {
  return c.x + dx * (c.y + dx * c.z);
}
template <class C, class T>
__device__ __forceinline__ T dspl_val(const C& c, T dx) {
  return c.w + dx * (c.x + dx * (T(0.5) * c.y + dx * (c.z * T(1.0 / 3.0))));
}

template <class T>
__device__ __forceinline__ typename V4<T>::type ldv4(const typename V4<T>::type* p);
template <>
__device__ __forceinline__ double4 ldv4<double>(const double4* p) {
  return ld_d4(p);
}
template <>
__device__ __forceinline__ float4 ldv4<float>(const float4* p) {
  return ld_keep(p);
}

// Both force rows of a single-type FP32 bin, (rho'_t) then (phi'), 32 bytes
// on a 32-byte boundary (one sector), in one 256-bit load: one L1 request per
// pair instead of two.
__device__ __forceinline__ void ld_rows2(const float4* p, float4& a, float4& b) {
  asm volatile("ld.global.nc.L1::evict_last.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// The derivative coefficients of one single-type FP64 bin from the two split
// arrays (the value slots stay unset).  A warp's 32 random bins cost 29 L1
// cycles this way, 49 as two 32-byte rows 64 bytes apart (which use half of
// the banks each), 32 as three 16-byte loads; the pass is bound by L1: EAM 131k
// FP64 6.47 -> 5.75 ms per 50 steps.
template <class T>
__device__ __forceinline__ void ld_derivs(const EamDev<T>& e, int idx, double4& rho,
                                          double4& phi) {
  rho = ld_d4(e.d4 + idx);
  phi.x = rho.w;
  asm volatile("ld.global.nc.L1::evict_last.v2.f64 {%0, %1}, [%2];"
      : "=d"(phi.y), "=d"(phi.z)
      : "l"(e.d2 + idx));
}

// Embedding F(rho), F'(rho) in FP64 (SplineTable eval/eval_deriv on F).
__device__ __forceinline__ void embed_eval(const double4* ftab, int nrho, double drho, int t,
                                           double rho, double& F, double& dF) {
  double dx;
  const int idx = spline_idx(rho, drho, nrho, dx);
  const double4 c = ldv4<double>(ftab + static_cast<long long>(t) * (nrho - 1) + idx);
  F = spl_val(c, dx);
  dF = spl_der(c, dx);
}

// Pass 1 (+ fused pass 2): rho_i = sum_j f_tj(r_ij); then fp_i = F'(rho_i)
// and, with EV, the embedding energy F(rho_i) into the block partials.
// types == nullptr means a single-type alloy.  gout (GeoQ only, nullable)
// receives the force pass's gather records {qx, qy, qz, bits(F'(rho))}.
template <class Geo, int LPA, int U, bool EV, bool VEC, bool MULTI, class FP, bool WIDE = false>
__global__ void __launch_bounds__(256) k_eam_density(Geo g, NbrView nl, int n,
                                                     EamDev<typename Geo::T> e,
                                                     const int* __restrict__ types,
                                                     FP* __restrict__ fp_out,
                                                     double* __restrict__ rho_out,
                                                     double* __restrict__ fpd_out,
                                                     int4* __restrict__ gout,
                                                     double* __restrict__ partials,
                                                     double* __restrict__ e_out,
                                                     double4* __restrict__ gout64) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA;
  const int sub = tid % LPA;
  const bool active = i < n;
  Acc<T> rho;
  typename Geo::Own o{};
  if (active) {
    o = g.own(i);
    const long long row = nl.row(i);
    const int c = nl.count(i);
    for (int base = first_slot<VEC, LPA, T, U>(sub); base < c; base += U * LPA) {
      int jj[U];
      nbr_batch<VEC, LPA, T>(nl, row, base, c, jj);
      typename Geo::Pair pr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (jj[u] >= 0)
          g.pair(o, jj[u], pr[u]);
        else
          pr[u].r2 = e.rc_sq;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (pr[u].r2 < e.rc_sq) {
          // No FP64-refined radius here: in the mixed path the density's
          // FP32 radius error is a few percent of the total force error
          // (the force pass's radius dominates), so it is not worth the
          // FP64 work.
          T sx;
          const int idx = spline_fast<WIDE>(g.radius_fast(pr[u]), e, sx);
          // fixed-point position records carry the atom's 1-based type in
          // their fourth word (the density pass always reads those)
          int tj = 0;
          if constexpr (MULTI) {
            if constexpr (Geo::kRecords)
              tj = pr[u].w - 1;
            else
              tj = __ldg(types + jj[u]) - 1;
          }
          const auto cf = ldv4<T>(e.dtab + static_cast<long long>(idx) * e.ntypes + tj);
          rho.add(spl_val(cf, sx));
        }
      }
    }
  }
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) rho.shfl_merge(s);
  double Fi = 0.0;
  if (active && sub == 0) {
    const double rh = rho.value();
    const int ti = MULTI ? __ldg(types + i) - 1 : 0;
    double dF;
    embed_eval(e.ftab, e.nrho, e.drho, ti, rh, Fi, dF);
    fp_out[i] = static_cast<FP>(dF);
    if (rho_out) rho_out[i] = rh;
    if (fpd_out) fpd_out[i] = dF;
    if (e_out) e_out[i] = Fi;
    if constexpr (has_d4out<Geo>::value) {
      if (gout64) gout64[i] = make_double4(o.x, o.y, o.z, dF);
    }
    if constexpr (Geo::kRecords) {
      if (gout) {
        int4 rec = g.record(o);
        rec.w = __float_as_int(static_cast<float>(dF));
        if (MULTI && e.tbits) {
          const int mask = (1 << e.tbits) - 1;
          rec.w = (rec.w & ~mask) | ti;
        }
        gout[i] = rec;
      }
    }
  }
  if (EV && partials) {
    const double w[6] = {0, 0, 0, 0, 0, 0};
    write_ev_partials(Fi, w, partials);
  }
}

// Pass 3: f_ij = -(phi' + fp_i rho'_tj + fp_j rho'_ti)/r * (r_i - r_j).
// FPG: F'(rho_j) comes with the neighbor's gather record (pair w bits)
// instead of the fp array.  KD (FPG, float forces): then the next step's
// kick + drift of the same atom.
template <class Geo, int LPA, int U, int EV, bool FPG, bool VEC, bool MULTI, class FP, class F,
          bool KD = false, bool WIDE = false>
__global__ void __launch_bounds__(256) k_eam_force(Geo g, NbrView nl, int n,
                                                   EamDev<typename Geo::T> e,
                                                   const int* __restrict__ types,
                                                   const FP* __restrict__ fp, ForceOut<F> out,
                                                   double* __restrict__ partials,
                                                   KickDrift kd = {},
                                                   double* __restrict__ pe_atom = nullptr) {
  dependent_launch_prologue();
  using T = typename Geo::T;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / LPA;
  const int sub = tid % LPA;
  const bool active = i < n;
  Acc<T> fx, fy, fz;
  double pe = 0.0;
  double w[6] = {0, 0, 0, 0, 0, 0};
  if (active) {
    const typename Geo::Own o = g.own(i);
    const long long row = nl.row(i);
    const int c = nl.count(i);
    const int ti = MULTI ? __ldg(types + i) - 1 : 0;
    // packed types (FPG, multi-type): F' of both atoms from the records with
    // the type bits cleared, so the pair term stays symmetric
    const bool packed = FPG && MULTI && e.tbits > 0;
    const int tmask = packed ? (1 << e.tbits) - 1 : 0;
    T fpi;
    if constexpr (FPG && MULTI && Geo::kRecords)
      fpi = packed ? __int_as_float(g.record(o).w & ~tmask) : static_cast<T>(__ldg(fp + i));
    else
      fpi = static_cast<T>(__ldg(fp + i));
    for (int base = first_slot<VEC, LPA, T, U>(sub); base < c; base += U * LPA) {
      int jj[U];
      nbr_batch<VEC, LPA, T>(nl, row, base, c, jj);
      typename Geo::Pair pr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (jj[u] >= 0)
          g.pair(o, jj[u], pr[u]);
        else
          pr[u].r2 = e.rc_sq;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (pr[u].r2 < e.rc_sq) {
          T r, rinv, corr, sx;
          g.radius2(o, pr[u], r, rinv, corr);
          const int idx = spline_at<WIDE>(r, corr, e, sx);
          const int j = jj[u];
          int tj = 0;
          if constexpr (MULTI && FPG && Geo::kRecords)
            tj = packed ? (pr[u].w & tmask) : __ldg(types + j) - 1;
          else if constexpr (MULTI)
            tj = __ldg(types + j) - 1;
          const auto* rowp = e.rtab + static_cast<long long>(idx) * e.S;
          typename V4<T>::type cphi, crho;
          if constexpr (!MULTI && sizeof(T) == sizeof(float)) {
            ld_rows2(rowp, crho, cphi);  // single type: S = 2, slots rho', phi'
          } else if constexpr (!MULTI) {
            ld_derivs(e, idx, crho, cphi);
            if (EV) cphi.w = __ldg(e.da + idx);
          } else {
            cphi = ldv4<T>(rowp + (MULTI ? phi_slot(ti, tj, e.ntypes) : 1));
            crho = ldv4<T>(rowp + tj);
          }
          const T drj = dspl_der(crho, sx);
          T dri = drj;
          if (MULTI && tj != ti) dri = dspl_der(ldv4<T>(rowp + ti), sx);
          T fpj;
          if constexpr (FPG) {
            fpj = g.gather_fp(pr[u], tmask);
          } else {
            fpj = static_cast<T>(__ldg(fp + j));
          }
          const T fpair = -div_r(dspl_der(cphi, sx) + fpi * drj + fpj * dri, r, rinv);
          fx.add(mul_rn(fpair, pr[u].dx));
          fy.add(mul_rn(fpair, pr[u].dy));
          fz.add(mul_rn(fpair, pr[u].dz));
          if (EV) {
            pe += 0.5 * static_cast<double>(dspl_val(cphi, sx));
            if (EV == 1) add_virial(w, fpair, pr[u].dx, pr[u].dy, pr[u].dz);
          }
        }
      }
    }
  }
#pragma unroll
  for (int s = LPA / 2; s > 0; s >>= 1) {
    fx.shfl_merge(s);
    fy.shfl_merge(s);
    fz.shfl_merge(s);
  }
  if (active && sub == 0) {
    out.store(i, fx.value(), fy.value(), fz.value());
    if constexpr (KD) {
      static_assert(FPG, "fused kick-drift: a force pass that reads gather records");
      kick_drift_atom<false>(kd, i, static_cast<F>(fx.value()), static_cast<F>(fy.value()),
                      static_cast<F>(fz.value()));
    }
  }
  if (KD && kd.step && blockIdx.x == 0 && threadIdx.x == 0) *kd.step += 1;
  if (EV) {
    // per-atom energy (nullable): the lanes' pair sums merged pairwise, plus
    // the embedding energy F(rho_i) the density pass stored there
    if (pe_atom) {
      double pa = pe;
#pragma unroll
      for (int o = LPA / 2; o > 0; o >>= 1) pa += __shfl_xor_sync(0xffffffffu, pa, o);
      if (active && sub == 0) pe_atom[i] = pa + pe_atom[i];
    }
    if (EV == 1 && partials) write_ev_partials(pe, w, partials);
  }
}

// Sums nblk partial records (kEvStride doubles each) in block order and
// ADDS them to energy[0] / virial[0..5] (either may be null).
__global__ void k_reduce_partials(const double* __restrict__ partials, int nblk,
                                  double* __restrict__ energy, double* __restrict__ virial);

// Threads of that one block: the records are a serial chain of loads per
// thread, so more than 512 records take 1024 threads (2530 records: 8.5 us
// with 256).
inline int reduce_threads(int nblk) { return nblk > 512 ? 1024 : 256; }

int force_blocks(long long n, int lpa);

}  // namespace tdmd_b200
