// su2_kernels.cuh -- device kernels of the checkerboard update sweep, the
// measurement reductions and the gradient flow, templated on the field
// precision R (double: plain FP64 path, float: precision form with FP64
// reductions) and on the field content CC (a compile-time content mask, or
// C_GENERIC to read it at run time).
//
// One thread owns one site of the parity being updated.  Sites of one parity
// never read each other's updated field (checkerboard), so a half-sweep is
// one launch, exactly as the reference's sequential site loop over that
// parity (update.c:35-259).
#pragma once

#include "su2_common.cuh"
#include "su2_launch.cuh"

namespace su2 {

#define HAS(bit) SU2_HAS(CC, cp.content, bit)
#define NHIGGS (HAS(C_H2) ? 2 : (HAS(C_H1) ? 1 : 0))

constexpr int BLOCK = 128;
// resident blocks per SM asked of the compiler: 8 x 128 threads caps FP32
// kernels at 64 registers (half occupancy); FP64 ones at 128
template <typename R>
struct MinBlocks {
  static constexpr int value = sizeof(R) == 4 ? 8 : 4;
};

// launch shapes of the update kernels the autotuner chooses from:
// (threads per block, resident blocks per SM asked of the compiler, which
// sets the register budget: 65536 / (threads * blocks))
constexpr int NVARIANTS = 4;
template <typename R, int V>
struct Variant;
template <typename R> struct Variant<R, 0> { static constexpr int BS = 128, MINB = sizeof(R) == 4 ? 8 : 4; };
template <typename R> struct Variant<R, 1> { static constexpr int BS = 128, MINB = sizeof(R) == 4 ? 5 : 3; };
template <typename R> struct Variant<R, 2> { static constexpr int BS = 256, MINB = sizeof(R) == 4 ? 4 : 2; };
template <typename R> struct Variant<R, 3> { static constexpr int BS = 64, MINB = sizeof(R) == 4 ? 12 : 6; };
// threads per block of each variant, for host code that builds tile tables
constexpr int kVariantBS[NVARIANTS] = {128, 128, 256, 64};
constexpr int NSUMS = 24;

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
// A lattice's counters are kept in CTR_COPIES copies of CTR_STRIDE words and
// summed when they are read: one atomic per warp on one address is a serial
// chain in L2 (measured 1.1 per ns), as long as a 128^3 lattice's pass itself.
// The chains of a pool have counters of their own, which spreads the atomics
// already; copies there only cost their address (384-chain ensemble: 2 %).
constexpr int CTR_COPIES = 16, CTR_STRIDE = 32;
constexpr size_t CTR_BYTES = (size_t)CTR_COPIES * CTR_STRIDE * 8;
__device__ inline unsigned long long* ctr_copy(unsigned long long* ctr, unsigned block) {
  return ctr + (block & (CTR_COPIES - 1)) * CTR_STRIDE;
}
__device__ inline void warp_count(unsigned long long* ctr, int v) {
  // every lane of the warp reaches this call (no early returns in kernels)
  int s = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(ctr, (unsigned long long)s);
}

// sum of v over the block, result valid in thread 0; blockDim.x <= 1024
__device__ inline double block_sum(double v) {
  __shared__ double sm[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[w] = v;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  if (w == 0) {
    v = lane < nw ? sm[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// ---------------------------------------------------------------------------
// SU(2) gauge part
// ---------------------------------------------------------------------------
// su2staple_wilson (staples.c:84-115)
template <typename R, bool RO = RO_DEFAULT>
__device__ inline Q<R> wilson_staple(const Fields<R>& f, const Geom& g, const int* c, int i, int mu) {
  Q<R> tot{(R)0, (R)0, (R)0, (R)0};
  int xp = shifted(g, c, mu, 1);
#pragma unroll
  for (int nu = 0; nu < 3; nu++) {
    if (nu == mu) continue;
    int xn = shifted(g, c, nu, 1);
    int xpm = shifted(g, c, mu, 1, nu, -1);
    int xm = shifted(g, c, nu, -1);
    Q<R> up = qmul(qmul(ldro4<R, RO>(lk(f, nu), xp), qdag(ldro4<R, RO>(lk(f, mu), xn))), qdag(ldro4<R, RO>(lk(f, nu), i)));
    tot = qadd(tot, up);
    Q<R> lo = qmul(qmul(qdag(ldro4<R, RO>(lk(f, nu), xpm)), qdag(ldro4<R, RO>(lk(f, mu), xm))), ldro4<R, RO>(lk(f, nu), xm));
    tot = qadd(tot, lo);
  }
  return tot;
}

// hopping_triplet_forward (su2u1.c:605-617): -Sigma(x) . R(U_mu(x)) Sigma(x+mu)
template <typename R>
__device__ inline R hop_triplet_fwd_u(const Fields<R>& f, const Geom& g, const int* c, int i, int mu,
                                      const Q<R>& U) {
  V3<R> r = qrot(U, ldro3(f, shifted(g, c, mu, 1)));
  return -dot3(ld3(f, i), r);
}

// su2link_staple (staples.c:134-193)
template <typename R, int CC>
__device__ inline Q<R> link_staple(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                   int mu) {
  Q<R> V = qscale(wilson_staple(f, g, c, i, mu), (R)-0.5 * cp.beta);
  const int nh = NHIGGS;
  if (nh > 0) {
    int xp = shifted(g, c, mu, 1);
    for (int h = 0; h < nh; h++) {
      Q<R> nphi = ldro4<R>(php(f, h), xp);
      if (HAS(C_U1)) {
        if constexpr (sizeof(R) == 8) nphi = qphase(nphi, a1p(f, mu)[i]);
        else nphi = qmul(nphi, u1phase(a1p(f, mu)[i]));
      }
      Q<R> t = qmul(nphi, qdag(ldro4<R>(php(f, h), i)));
      V.a -= (R)0.5 * t.a;
      V.b -= (R)0.5 * t.b;
      V.c -= (R)0.5 * t.c;
      V.d -= (R)0.5 * t.d;
    }
  }
  return V;
}

// su2ptrace (su2u1.c:108-116) at site x (index i, coords c)
template <typename R>
__device__ inline R ptrace(const Fields<R>& f, const Geom& g, const int* c, int i, int mu, int nu) {
  Q<R> s = qmul(qmul(ld4<R>(lk(f, mu), i), ld4<R>(lk(f, nu), shifted(g, c, mu, 1))),
                qdag(ld4<R>(lk(f, mu), shifted(g, c, nu, 1))));
  return (R)2 * qdot0(s, qdag(ld4<R>(lk(f, nu), i)));
}

// ---------------------------------------------------------------------------
// doublet
// ---------------------------------------------------------------------------
template <typename R>
__device__ inline R doubletsq(const Q<R>& a) {
  return (R)0.5 * (a.a * a.a + a.b * a.b + a.c * a.c + a.d * a.d);
}
template <typename R>
__device__ inline R tripletsq(const V3<R>& a) {
  return (R)0.5 * (a.x * a.x + a.y * a.y + a.z * a.z);
}

// hopping_trace(_su2u1) (su2u1.c:388-418): Re Tr Phi1^+ U Phi2 e^{-i a s3}
template <typename R, int CC>
__device__ inline R hop_trace(const CoupT<R>& cp, const Q<R>& p1, const Q<R>& u, const Q<R>& p2, R alpha) {
  Q<R> t = qmul(u, p2);
  if (HAS(C_U1)) {
    if constexpr (sizeof(R) == 8) t = qphase(t, alpha);
    else t = qmul(t, u1phase(alpha));
  }
  return qdot0(qdag(p1), t);
}
template <typename R, int CC>
__device__ inline R hop_doublet_fwd(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    int mu, int h) {
  R al = HAS(C_U1) ? a1p(f, mu)[i] : (R)0;
  return -hop_trace<R, CC>(cp, ld4<R>(php(f, h), i), ld4<R>(lk(f, mu), i), ld4<R>(php(f, h), shifted(g, c, mu, 1)), al);
}
template <typename R, int CC>
__device__ inline R hop_doublet_bwd(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    int mu, int h) {
  int pm = shifted(g, c, mu, -1);
  R al = HAS(C_U1) ? a1p(f, mu)[pm] : (R)0;
  return -hop_trace<R, CC>(cp, ld4<R>(php(f, h), pm), ld4<R>(lk(f, mu), pm), ld4<R>(php(f, h), i), al);
}
template <typename R, int CC>
__device__ inline R covariant_doublet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                      int h) {
  R tot = 0, mod = doubletsq(ld4<R>(php(f, h), i));
#pragma unroll
  for (int d = 0; d < 3; d++) tot += (R)2 * mod + hop_doublet_fwd<R, CC>(f, g, cp, c, i, d, h);
  return tot;
}

// potential_singlet (su2u1.c:708-723)
template <typename R, int CC>
__device__ inline R potential_singlet(const Fields<R>& f, const CoupT<R>& cp, int i) {
  R S = f.sing[i];
  R pot = (R)cp.b1s * S + (R)0.5 * (R)cp.msqs * S * S + (R)(1.0 / 3.0) * (R)cp.b3s * S * S * S +
          (R)0.25 * (R)cp.b4s * S * S * S * S;
  if (NHIGGS == 1) {
    R mod = doubletsq(ld4<R>(php(f, 0), i));
    pot += (R)0.5 * (R)cp.a1s * S * mod + (R)0.5 * (R)cp.a2s * S * S * mod;
  }
  return pot;
}

// higgspotential (su2u1.c:528-572)
template <typename R, int CC>
__device__ inline R higgspotential(const Fields<R>& f, const CoupT<R>& cp, int i) {
  R pot = 0, mod = 0;
  const int nh = NHIGGS;
  if (nh > 0) {
    Q<R> h1 = ld4<R>(php(f, 0), i);
    mod = doubletsq(h1);
    pot += (R)cp.msq * mod + (R)cp.lam * mod * mod;
    if (nh == 2) {
      Q<R> h2 = ld4<R>(php(f, 1), i);
      R f11 = mod, f22 = doubletsq(h2);
      R Re = (R)0.5 * (h1.a * h2.a + h1.b * h2.b + h1.c * h2.c + h1.d * h2.d);
      R Im = (R)0.5 * (h1.d * h2.a + h1.c * h2.b - h1.b * h2.c - h1.a * h2.d);
      pot += (R)cp.msq2 * f22 + (R)cp.m12re * Re - (R)cp.m12im * Im + (R)cp.lam2 * f22 * f22 +
             (R)cp.lam3 * f11 * f22 + (R)cp.lam4 * (Re * Re + Im * Im) + (R)cp.lam5re * (Re * Re - Im * Im) -
             (R)2 * (R)cp.lam5im * Re * Im + f11 * ((R)cp.lam6re * Re - (R)cp.lam6im * Im) +
             f22 * ((R)cp.lam7re * Re + (R)cp.lam7im * Im);
    }
  }
  if (HAS(C_T)) {
    R mt = tripletsq(ld3(f, i));
    pot += (R)cp.msqT * mt + (R)cp.b4 * mt * mt;
    if (nh > 0) pot += (R)cp.a2 * mod * mt;
  }
  if (HAS(C_S)) pot += potential_singlet<R, CC>(f, cp, i);
  return pot;
}

// localact_doublet (su2u1.c:495-510)
template <typename R, int CC>
__device__ inline R localact_doublet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                     int h) {
  R tot = covariant_doublet<R, CC>(f, g, cp, c, i, h);
#pragma unroll
  for (int d = 0; d < 3; d++) tot += hop_doublet_bwd<R, CC>(f, g, cp, c, i, d, h);
  tot += higgspotential<R, CC>(f, cp, i);
  return tot;
}

// staple_doublet (staples.c:243-302)
template <typename R, int CC>
__device__ inline Q<R> staple_doublet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                      int h) {
  Q<R> res{(R)0, (R)0, (R)0, (R)0};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    int xp = shifted(g, c, d, 1), xm = shifted(g, c, d, -1);
    Q<R> w = qmul(ldro4<R>(lk(f, d), i), ldro4<R>(php(f, h), xp));
    if (HAS(C_U1)) {
      if constexpr (sizeof(R) == 8) w = qphase(w, a1p(f, d)[i]);
      else w = qmul(w, u1phase(a1p(f, d)[i]));
    }
    res.a -= w.a; res.b -= w.b; res.c -= w.c; res.d -= w.d;
    w = qmul(qdag(ldro4<R>(lk(f, d), xm)), ldro4<R>(php(f, h), xm));
    if (HAS(C_U1)) {
      if constexpr (sizeof(R) == 8) w = qphase(w, -a1p(f, d)[xm]);
      else w = qmul(w, qdag(u1phase(a1p(f, d)[xm])));
    }
    res.a -= w.a; res.b -= w.b; res.c -= w.c; res.d -= w.d;
  }
  return res;
}

// ---------------------------------------------------------------------------
// triplet
// ---------------------------------------------------------------------------
template <typename R>
__device__ inline R hop_triplet_fwd(const Fields<R>& f, const Geom& g, const int* c, int i, int mu) {
  return hop_triplet_fwd_u(f, g, c, i, mu, ld4<R>(lk(f, mu), i));
}
template <typename R>
__device__ inline R covariant_triplet(const Fields<R>& f, const Geom& g, const int* c, int i) {
  R tot = 0, mod = tripletsq(ld3(f, i));
#pragma unroll
  for (int d = 0; d < 3; d++) tot += (R)2 * mod + hop_triplet_fwd(f, g, c, i, d);
  return tot;
}

// localact_su2link (su2u1.c:166-198)
template <typename R, int CC>
__device__ inline R localact_su2link(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                     int mu) {
  R tot = 0;
#pragma unroll
  for (int nu = 0; nu < 3; nu++) {
    if (nu == mu) continue;
    tot += ((R)1 - (R)0.5 * ptrace(f, g, c, i, mu, nu));
    int cm[3];
    shift_coords(g, c, nu, -1, cm);
    tot += ((R)1 - (R)0.5 * ptrace(f, g, cm, shifted(g, c, nu, -1), mu, nu));
  }
  tot *= (R)cp.beta;
  for (int h = 0; h < NHIGGS; h++) tot += hop_doublet_fwd<R, CC>(f, g, cp, c, i, mu, h);
  if (HAS(C_T)) tot += hop_triplet_fwd(f, g, c, i, mu);
  return tot;
}

// ---------------------------------------------------------------------------
// U(1)
// ---------------------------------------------------------------------------
template <typename R>
__device__ inline R u1ptrace(const Fields<R>& f, const Geom& g, const int* c, int i, int d1, int d2) {
  return a1p(f, d1)[i] + a1p(f, d2)[shifted(g, c, d1, 1)] - a1p(f, d1)[shifted(g, c, d2, 1)] - a1p(f, d2)[i];
}
// local_u1wilson (su2u1.c:316-328)
template <typename R>
__device__ inline R local_u1wilson(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i) {
  R res = 0;
#pragma unroll
  for (int d1 = 0; d1 < 3; d1++)
#pragma unroll
    for (int d2 = 0; d2 < d1; d2++) res += ((R)1 - mcos((R)cp.r_u1 * u1ptrace(f, g, c, i, d2, d1)));
  return (R)cp.betau1 * res;
}
// localact_u1link (su2u1.c:336-354)
template <typename R, int CC>
__device__ inline R localact_u1link(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    int mu) {
  R tot = 0;
#pragma unroll
  for (int nu = 0; nu < 3; nu++) {
    if (nu == mu) continue;
    tot += ((R)1 - mcos((R)cp.r_u1 * u1ptrace(f, g, c, i, mu, nu)));
    int cm[3];
    shift_coords(g, c, nu, -1, cm);
    tot += ((R)1 - mcos((R)cp.r_u1 * u1ptrace(f, g, cm, shifted(g, c, nu, -1), mu, nu)));
  }
  tot *= (R)cp.betau1;
  for (int h = 0; h < NHIGGS; h++) tot += hop_doublet_fwd<R, CC>(f, g, cp, c, i, mu, h);
  return tot;
}

// ---------------------------------------------------------------------------
// real root of a x^3 + b x^2 + c x + d (polysolve3, overrelax.c:14-34):
// Cardano's formula followed by Newton steps on the cubic.  The reference
// evaluates Cardano's formula in long double: the leading coefficient of
// these cubics is lambda/4 (~5e-4), so the formula cancels, and in double it
// lands up to ~1e-11 away (relative) from the long-double root.  The cubic
// itself is well conditioned near its root (the linear coefficient
// dominates), so Newton steps bring the result to the root within rounding,
// matching the reference's long-double value to ~1e-15.
// FP32: two Newton steps.  FP64: since the Newton steps, not the formula, fix
// the accuracy, the start comes from the FP32 root, and the steps multiply by
// an FP32 reciprocal of the slope: the first leaves ~1e-12 of the root's
// scale, the second rounding.  FP64 Cardano (a square root, a cube root, two
// divisions, ~95 FP64 instructions, each holding a quarter's pipe 64 cycles) stays
// for the cubics where that start is no good: FP32 has no root of its own, the
// slope is beyond FP32 (its reciprocal would be 0 and a correction of 0 mean
// nothing), or the last correction is above 1e-10 of the root.
// ---------------------------------------------------------------------------
__device__ inline double polysolve3_f64(double a, double b, double c, double d, int* fallback);
template <typename R>
__device__ inline R polysolve3(R a, R b, R c, R d, int* fallback) {
  if constexpr (sizeof(R) == 8) return polysolve3_f64(a, b, c, d, fallback);
  R discr = (R)18 * a * b * c * d - (R)4 * b * b * b * d + b * b * c * c - (R)4 * a * c * c * c - (R)27 * a * a * d * d;
  R del1 = (R)2 * b * b * b - (R)9 * a * b * c + (R)27 * a * a * d;
  R x;
  if (discr < (R)0) {
    R A = (R)0.5 * (del1 + a * msqrt((R)(-27) * discr));
    A = mcbrt(A);
    x = -(b + A + (b * b - (R)3 * a * c) / A) / ((R)3 * a);
#pragma unroll
    for (int it = 0; it < 2; it++) {
      R fx = ((a * x + b) * x + c) * x + d;
      R dfx = ((R)3 * a * x + (R)2 * b) * x + c;
      x -= fx / dfx;
    }
  } else {
    x = b / a;
    *fallback = 1;
  }
  return x;
}
// one Newton step with the slope's reciprocal in FP32; whether that slope is in
// FP32's range, and the correction
__device__ inline bool newton3(double a, double b, double c, double d, double* x, double* dx) {
  const double fx = fma(fma(fma(a, *x, b), *x, c), *x, d);
  const double dfx = fma(fma(3.0 * a, *x, 2.0 * b), *x, c);
  *dx = fx * (double)(1.0f / (float)dfx);
  *x -= *dx;
  return fabs(dfx) < 1e37;
}
__device__ inline double polysolve3_f64(double a, double b, double c, double d, int* fallback) {
  const double discr = 18.0 * a * b * c * d - 4.0 * b * b * b * d + b * b * c * c - 4.0 * a * c * c * c - 27.0 * a * a * d * d;
  if (!(discr < 0.0)) {
    *fallback = 1;
    return b / a;
  }
  int fb = 0;
  double x = (double)polysolve3<float>((float)a, (float)b, (float)c, (float)d, &fb), dx;
  newton3(a, b, c, d, &x, &dx);
  const bool in_range = newton3(a, b, c, d, &x, &dx);
  // an FP32 root of another branch or a NaN fails the last test
  if (fb || !in_range || !(fabs(dx) <= 1e-10 * fabs(x))) {
    const double del1 = 2.0 * b * b * b - 9.0 * a * b * c + 27.0 * a * a * d;
    const double A = cbrt(0.5 * (del1 + a * sqrt(-27.0 * discr)));
    x = -(b + A + (b * b - 3.0 * a * c) / A) / (3.0 * a);
    const double fx = ((a * x + b) * x + c) * x + d;
    x -= fx / ((3.0 * a * x + 2.0 * b) * x + c);
  }
  return x;
}
// ---------------------------------------------------------------------------
// local updates.  The overrelaxation updates take their random-number source
// as a template parameter: the sweep kernels pass the site's stream
// (SiteRng), the per-site verification kernel ZeroRng, whose uniforms are
// all 0, so that every proposal is accepted and can be read back.
// ---------------------------------------------------------------------------
template <typename R>
struct ZeroRng {
  __device__ R uni() { return (R)0; }
};
// heatbath_su2link (heatbath.c:15-124): Kennedy-Pendleton; the uniforms are
// drawn in the reference's order (4 per trial, 3 per sphere trial, 1 for the
// triplet accept/reject).  The first trial's four are drawn before the staple
// is gathered: the same values in the same order (each site's stream is
// positional), with the generator's arithmetic free to run while the loads
// are in flight.  The other local updates draw early in the same way.
template <typename R, int CC>
__device__ inline int heatbath(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i, int mu,
                               SiteRng<R>& rng, int* kpcap, int* err) {
  R u0 = rng.uni(), u1 = rng.uni(), u2 = rng.uni(), u3 = rng.uni();  // the first trial's
  Q<R> old{};
  R oldact = 0;
  if (HAS(C_T)) {
    old = ld4<R>(lk(f, mu), i);
    oldact = hop_triplet_fwd_u(f, g, c, i, mu, old);
  }
  Q<R> V = link_staple<R, CC>(f, g, cp, c, i, mu);
  R a = 0, ia = 0;  // FP64 uses ia = 1 / (2 |V|), one reciprocal square root
  if constexpr (sizeof(R) == 8) {
    ia = rsqrt(qsq(V));
    V = qscale(V, -ia);
    ia *= (R)0.5;
  } else {
    a = msqrt(qsq(V));
    V = qscale(V, (R)-1 / a);
    a *= (R)2;
  }
  R a0, r1, r2, r3, d;
  int loop = 1;
  do {
    if (loop > 1) {
      u0 = rng.uni();
      u1 = rng.uni();
      u2 = rng.uni();
      u3 = rng.uni();
    }
    if constexpr (sizeof(R) == 8) {
      r1 = -mlog((R)1 - u0) * ia;
      r2 = -mlog((R)1 - u1) * ia;
    } else {
      r1 = -mlog((R)1 - u0) / a;
      r2 = -mlog((R)1 - u1) / a;
    }
    r3 = mcos2pi(u2);
    r3 *= r3;
    d = r1 * r3 + r2;
    r3 = (R)1 - u3;
    loop++;
  } while (r3 * r3 > (R)1 - (R)0.5 * d && loop <= 200);
  R rad;
  if (loop > 200) {
    a0 = (R)1e-9;
    *kpcap = 1;
    rad = (R)1 - a0 * a0;
  } else {
    a0 = (R)1 - d;
    // FP32: 1 - a0^2 = d (2 - d) without the cancellation near a0 = 1
    rad = sizeof(R) == 8 ? (R)1 - a0 * a0 : d * ((R)2 - d);
  }
  if (rad < (R)0) return 0;
  rad = msqrt(rad);
  Q<R> nl;
  if constexpr (sizeof(R) == 8) {
    // uniform direction on S^2 by rejection from the cube (heatbath.c:82-93)
    d = 2;
    int it = 0;
    while (d > (R)1 || d == (R)0) {
      r1 = (R)2 * rng.uni() - (R)1;
      r2 = (R)2 * rng.uni() - (R)1;
      r3 = (R)2 * rng.uni() - (R)1;
      d = r1 * r1 + r2 * r2 + r3 * r3;
      if (++it > 4096) {  // probability (1 - pi/6)^4096: never; guards a NaN state
        *err = 1;
        return 0;
      }
    }
    d = rad * rsqrt(d);
    nl = Q<R>{a0, r1 * d, r2 * d, r3 * d};
  } else {
    // FP32 form: the same uniform direction drawn directly (Archimedes:
    // cos(theta) uniform on [-1,1], azimuth uniform), no rejection loop to
    // diverge a warp
    float z = 2.0f * rng.uni() - 1.0f;
    float ph = rng.uni();
    float sn, cs;
    sincospif(2.0f * ph, &sn, &cs);
    float s = sqrtf(fmaxf(0.0f, 1.0f - z * z)) * rad;
    nl = Q<R>{a0, s * cs, s * sn, z * rad};
  }
  Q<R> U = unitize(qmul(nl, qdag(V)));
  st4<R>(lk(f, mu), i, U);
  if (HAS(C_T)) {
    R diff = oldact - hop_triplet_fwd_u(f, g, c, i, mu, U);
    if (rng.uni() < mexp(diff)) return 1;
    st4<R>(lk(f, mu), i, old);
    return 0;
  }
  return 1;
}

// FP32 form: every link written is re-normalised to unit length, so rounding
// never accumulates in the SU(2) constraint (the FP64 path writes the product
// as it is, as the reference does)
template <typename R>
__device__ inline Q<R> unitize(const Q<R>& q) {
  if (sizeof(R) == 8) return q;
  return qscale(q, (R)rsqrtf((float)qsq(q)));
}

// Metropolis decision (metropolis.c:15-167)
template <typename R>
__device__ inline int metro_accept(R diff, SiteRng<R>& rng) {
  if (diff < (R)0) return 1;
  if (diff > (R)0 && mexp(-diff) > rng.uni()) return 1;
  return 0;
}
// the same with the decision's uniform u drawn beforehand (it is the site's
// last draw of the pass, so drawing it whatever diff turns out to be changes
// no other draw)
template <typename R>
__device__ inline int metro_accept_u(R diff, R u) {
  if (diff < (R)0) return 1;
  if (diff > (R)0 && mexp(-diff) > u) return 1;
  return 0;
}

// metro_su2link (metropolis.c:15-41) with random_su2link (init.c:43-58)
template <typename R, int CC>
__device__ inline int metro_link(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i, int mu,
                                 SiteRng<R>& rng) {
  Q<R> old = ld4<R>(lk(f, mu), i);
  R a0 = localact_su2link<R, CC>(f, g, cp, c, i, mu);
  Q<R> u;
  u.a = (R)10 * (rng.uni() - (R)0.5);
  u.b = (R)1 * (rng.uni() - (R)0.5);
  u.c = (R)1 * (rng.uni() - (R)0.5);
  u.d = (R)1 * (rng.uni() - (R)0.5);
  R n = msqrt(u.a * u.a + u.b * u.b + u.c * u.c + u.d * u.d);
  u = Q<R>{u.a / n, u.b / n, u.c / n, u.d / n};
  st4<R>(lk(f, mu), i, unitize(qmul(old, u)));
  R a1 = localact_su2link<R, CC>(f, g, cp, c, i, mu);
  if (metro_accept(a1 - a0, rng)) return 1;
  st4<R>(lk(f, mu), i, old);
  return 0;
}

// The FP64 forms of the updates below, which the FP64 pipe bounds (2 lanes a
// cycle and SM; an OR pass of a 16^3 lattice spent 319 FP64 instructions per
// site, 16^3 sweep + measurement 325 -> 276 us with these): each update's
// action difference is formed once from the staple, and divided by once.

// metro_u1link (metropolis.c:48-70): the plaquettes' change from cos A -
// cos(A + e) = 2 sin(A + e/2) sin(e/2), five trigonometric functions instead
// of eight, and the hopping terms' from one gather
template <int CC>
__device__ inline int metro_u1_f64(const Fields<double>& f, const Geom& g, const CoupT<double>& cp, const int* c,
                                   int i, int mu, SiteRng<double>& rng) {
  using R = double;
  const R old = a1p(f, mu)[i], e = 0.95 * (rng.uni() - 0.5), eh = 0.5 * cp.r_u1 * e;
  R sum = 0;
#pragma unroll
  for (int nu = 0; nu < 3; nu++) {
    if (nu == mu) continue;
    // the link enters the plaquette at the site with +, the one below with -
    sum += sin(fma(cp.r_u1, u1ptrace(f, g, c, i, mu, nu), eh));
    int cm[3];
    shift_coords(g, c, nu, -1, cm);
    sum -= sin(fma(cp.r_u1, u1ptrace(f, g, cm, shifted(g, c, nu, -1), mu, nu), -eh));
  }
  R diff = 2.0 * cp.betau1 * sin(eh) * sum;
  const int xp = shifted(g, c, mu, 1);
  for (int h = 0; h < NHIGGS; h++) {
    const Q<R> p = qdag(ld4<R>(php(f, h), i)), t = qmul(ld4<R>(lk(f, mu), i), ld4<R>(php(f, h), xp));
    diff -= qdot0(p, qphase(t, old + e)) - qdot0(p, qphase(t, old));
  }
  if (!metro_accept(diff, rng)) return 0;
  a1p(f, mu)[i] = old + e;
  return 1;
}

// metro_doublet (metropolis.c:77-106): every hopping term is linear in the
// field, so dS = (p'-p).s + 3 (p'^2-p^2) + V(p') - V(p) with s =
// staple_doublet -- the neighbours are multiplied once instead of four times
template <int CC>
__device__ inline int metro_doublet_f64(const Fields<double>& f, const CoupT<double>& cp, int i, int h,
                                        const Q<double>& s, SiteRng<double>& rng) {
  using R = double;
  const R d0 = rng.uni() - 0.5, d1 = rng.uni() - 0.5, d2 = rng.uni() - 0.5, d3 = rng.uni() - 0.5;
  const Q<R> old = ld4<R>(php(f, h), i), nw{old.a + d0, old.b + d1, old.c + d2, old.d + d3};
  const Q<R> e{nw.a - old.a, nw.b - old.b, nw.c - old.c, nw.d - old.d};
  const R dsq = e.a * (nw.a + old.a) + e.b * (nw.b + old.b) + e.c * (nw.c + old.c) + e.d * (nw.d + old.d);
  const R v0 = higgspotential<R, CC>(f, cp, i);
  st4<R>(php(f, h), i, nw);
  const R diff = (e.a * s.a + e.b * s.b + e.c * s.c + e.d * s.d) + 3.0 * dsq + (higgspotential<R, CC>(f, cp, i) - v0);
  if (metro_accept(diff, rng)) return 1;
  st4<R>(php(f, h), i, old);
  return 0;
}

// |v| and v / |v| from v^2: CUDA's reciprocal root, and from it by one Newton step
// each the root and the direction, as exact as with sqrt and a division per
// component.  (|v| as v^2 rsqrt(v^2), and a direction by one reciprocal, cost the
// overrelaxation 12 % in rms error: 1.45 against 1.30 units of 2^-53; with these 1.20.)
template <int N>
__device__ inline double direction_f64(const double (&v)[N], double vsq, double (&e)[N]) {
  const double y = rsqrt(vsq), r = vsq * y, F = fma(0.5 * y, fma(-r, r, vsq), r), dy = y * fma(-F, y, 1.0);
#pragma unroll
  for (int k = 0; k < N; k++) e[k] = fma(v[k], dy, v[k] * y);
  return F;
}

// the overrelaxation of a field with N components p in the action p.s + B p^2
// + C p^4 (overrelax.c:54-236): p is replaced if u accepts the proposal
template <int N>
__device__ inline int overrelax_f64(double (&p)[N], const double (&s)[N], double B, double C, double u,
                                    int* fallback) {
  double ss = 0, e[N], X = 0, y[N], Ysq = 0;
#pragma unroll
  for (int k = 0; k < N; k++) ss += s[k] * s[k];
  const double F = direction_f64(s, ss, e);
#pragma unroll
  for (int k = 0; k < N; k++) X += p[k] * e[k];
#pragma unroll
  for (int k = 0; k < N; k++) {
    y[k] = p[k] - X * e[k];
    Ysq += y[k] * y[k];
  }
  // (V(x) - V(X)) / (x - X) = C x^3 + b x^2 + c x + d
  const double b = C * X, c = B + C * fma(X, X, 2.0 * Ysq);
  const double newX = polysolve3<double>(C, b, c, fma(c, X, F), fallback);
  const double dV = fma(fma(4.0 * C, fma(X, X, Ysq), 2.0 * B), X, F);
  const double dVn = fma(fma(4.0 * C, fma(newX, newX, Ysq), 2.0 * B), newX, F);
  if (!(fabs(dV) >= u * fabs(dVn))) return 0;
#pragma unroll
  for (int k = 0; k < N; k++) p[k] = newX * e[k] - y[k];
  return 1;
}

// the doublet's (one doublet) and the triplet's, with their staples s
template <int CC>
__device__ inline int overrelax_doublet_f64(const Fields<double>& f, const CoupT<double>& cp, int i,
                                            const Q<double>& s, double u, int* fallback) {
  const Q<double> p = ld4<double>(php(f, 0), i);
  double B = 0.5 * cp.msq + 3.0;
  if (HAS(C_T)) B += 0.5 * cp.a2 * tripletsq(ld3(f, i));
  if (HAS(C_S)) {
    const double S = f.sing[i];
    B += 0.25 * cp.a1s * S + 0.25 * cp.a2s * S * S;
  }
  const double sv[4] = {s.a, s.b, s.c, s.d};
  double pv[4] = {p.a, p.b, p.c, p.d};
  if (!overrelax_f64<4>(pv, sv, B, 0.25 * cp.lam, u, fallback)) return 0;
  st4<double>(php(f, 0), i, Q<double>{pv[0], pv[1], pv[2], pv[3]});
  return 1;
}
__device__ inline int overrelax_triplet_f64(const Fields<double>& f, const CoupT<double>& cp, int i,
                                            const V3<double>& s, double u, int* fallback) {
  const V3<double> t = ld3(f, i);
  const double sv[3] = {s.x, s.y, s.z};
  double tv[3] = {t.x, t.y, t.z};
  if (!overrelax_f64<3>(tv, sv, 0.5 * cp.msqT + 3.0, 0.25 * cp.b4, u, fallback)) return 0;
  st3(f, i, V3<double>{tv[0], tv[1], tv[2]});
  return 1;
}
// metro_triplet's FP64 form with its staple s (see metro_triplet)
template <int CC>
__device__ inline int metro_triplet_f64(const Fields<double>& f, const CoupT<double>& cp, int i, const V3<double>& s,
                                        SiteRng<double>& rng) {
  const double dx = rng.uni() - 0.5, dy = rng.uni() - 0.5, dz = rng.uni() - 0.5;
  const V3<double> old = ld3(f, i), nw{old.x + dx, old.y + dy, old.z + dz};
  const double ex = nw.x - old.x, ey = nw.y - old.y, ez = nw.z - old.z;
  const double dsq = ex * (nw.x + old.x) + ey * (nw.y + old.y) + ez * (nw.z + old.z);
  const double ssq = (nw.x * nw.x + nw.y * nw.y + nw.z * nw.z) + (old.x * old.x + old.y * old.y + old.z * old.z);
  double B = 0.5 * cp.msqT + 3.0;
  if (NHIGGS > 0) B += 0.5 * cp.a2 * doubletsq(ld4<double>(php(f, 0), i));
  if (!metro_accept(ex * s.x + ey * s.y + ez * s.z + dsq * (B + 0.25 * cp.b4 * ssq), rng)) return 0;
  st3(f, i, nw);
  return 1;
}

// metro_u1link (metropolis.c:48-70)
template <typename R, int CC>
__device__ inline int metro_u1(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i, int mu,
                               SiteRng<R>& rng) {
  if constexpr (sizeof(R) == 8) return metro_u1_f64<CC>(f, g, cp, c, i, mu, rng);
  R old = a1p(f, mu)[i];
  R a0 = localact_u1link<R, CC>(f, g, cp, c, i, mu);
  a1p(f, mu)[i] = old + (R)0.95 * (rng.uni() - (R)0.5);
  R a1 = localact_u1link<R, CC>(f, g, cp, c, i, mu);
  if (metro_accept(a1 - a0, rng)) return 1;
  a1p(f, mu)[i] = old;
  return 0;
}

// metro_doublet (metropolis.c:77-106)
template <typename R, int CC>
__device__ inline int metro_doublet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    int h, SiteRng<R>& rng) {
  if constexpr (sizeof(R) == 8)
    return metro_doublet_f64<CC>(f, cp, i, h, staple_doublet<R, CC>(f, g, cp, c, i, h), rng);
  const R d0 = rng.uni() - (R)0.5, d1 = rng.uni() - (R)0.5, d2 = rng.uni() - (R)0.5, d3 = rng.uni() - (R)0.5;
  Q<R> old = ld4<R>(php(f, h), i);
  R a0 = localact_doublet<R, CC>(f, g, cp, c, i, h);
  Q<R> nw = old;
  nw.a += (R)1 * d0;
  nw.b += (R)1 * d1;
  nw.c += (R)1 * d2;
  nw.d += (R)1 * d3;
  st4<R>(php(f, h), i, nw);
  R a1 = localact_doublet<R, CC>(f, g, cp, c, i, h);
  if (metro_accept(a1 - a0, rng)) return 1;
  st4<R>(php(f, h), i, old);
  return 0;
}

// overrelax_doublet (overrelax.c:54-128)
template <typename R, int CC, typename RNG>
__device__ inline int overrelax_doublet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                        RNG& rng, int* fallback) {
  const R u = rng.uni();
  if constexpr (sizeof(R) == 8)
    return overrelax_doublet_f64<CC>(f, cp, i, staple_doublet<R, CC>(f, g, cp, c, i, 0), u, fallback);
  Q<R> s = staple_doublet<R, CC>(f, g, cp, c, i, 0);
  Q<R> p = ld4<R>(php(f, 0), i);
  R F = msqrt(s.a * s.a + s.b * s.b + s.c * s.c + s.d * s.d);
  const R iF = (R)1 / F;  // one reciprocal instead of nine divisions
  R X = (p.a * s.a + p.b * s.b + p.c * s.c + p.d * s.d) * iF;
  R y0 = p.a - X * s.a * iF;
  R y1 = p.b - X * s.b * iF;
  R y2 = p.c - X * s.c * iF;
  R y3 = p.d - X * s.d * iF;
  R Ysq = y0 * y0 + y1 * y1 + y2 * y2 + y3 * y3;
  R B = (R)0.5 * (R)cp.msq + (R)3;
  if (HAS(C_T)) B += (R)0.5 * (R)cp.a2 * tripletsq(ld3(f, i));
  if (HAS(C_S)) {
    R S = f.sing[i];
    B += (R)0.25 * (R)cp.a1s * S + (R)0.25 * (R)cp.a2s * S * S;
  }
  R C = (R)0.25 * (R)cp.lam;
  R cc = B + (R)2 * Ysq * C;
  R newX = polysolve3<R>(C, C * X, cc + C * X * X, F + cc * X + C * X * X * X, fallback);
  R dV = F + (R)2 * B * X + (R)4 * C * (X * X * X + Ysq * X);
  R dVn = F + (R)2 * B * newX + (R)4 * C * (newX * newX * newX + Ysq * newX);
  if (mabs(dV / dVn) >= u) {
    R k = (newX + X);
    st4<R>(php(f, 0), i, Q<R>{-p.a + k * s.a * iF, -p.b + k * s.b * iF, -p.c + k * s.c * iF, -p.d + k * s.d * iF});
    return 1;
  }
  return 0;
}

// overrelax_higgs2 (overrelax.c:295-417)
template <typename R, int CC, typename RNG>
__device__ inline int overrelax_higgs2(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                       int h, RNG& rng, int* fallback, const Q<R>* given = nullptr) {
  const R u = rng.uni();
  Q<R> s;
  if constexpr (sizeof(R) == 8) s = given ? *given : staple_doublet<R, CC>(f, g, cp, c, i, h);
  else s = staple_doublet<R, CC>(f, g, cp, c, i, h);
  Q<R> fv = ld4<R>(php(f, h), i);
  Q<R> H;
  R l67re, l67im, lore, loim, lam12, msq;
  int sign;
  if (h == 0) {
    H = ld4<R>(php(f, 1), i);
    sign = -1;
    lam12 = cp.lam; msq = cp.msq;
    l67re = cp.lam7re; l67im = cp.lam7im; lore = cp.lam6re; loim = -cp.lam6im;
  } else {
    H = ld4<R>(php(f, 0), i);
    sign = 1;
    lam12 = cp.lam2; msq = cp.msq2;
    l67re = cp.lam6re; l67im = -cp.lam6im; lore = cp.lam7re; loim = cp.lam7im;
  }
  R Hv[4] = {H.a, H.b, H.c, H.d};
  R G[4] = {sign * Hv[3], sign * Hv[2], -(R)sign * Hv[1], -(R)sign * Hv[0]};
  R Hsq = doubletsq(H);
  R sv[4] = {s.a, s.b, s.c, s.d}, fr[4] = {fv.a, fv.b, fv.c, fv.d};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    sv[k] += (R)0.5 * ((R)cp.m12re + Hsq * l67re) * Hv[k];
    sv[k] += (R)0.5 * (-(R)cp.m12im + Hsq * l67im) * G[k];
    sv[k] = -sv[k];
  }
  R F = sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2] + sv[3] * sv[3];
  R X = 0;
  if constexpr (sizeof(R) == 8) {
    R e[4];
    F = direction_f64(sv, F, e);
#pragma unroll
    for (int k = 0; k < 4; k++) { sv[k] = e[k]; X += fr[k] * sv[k]; }
  } else {
    F = msqrt(F);
#pragma unroll
    for (int k = 0; k < 4; k++) { sv[k] /= F; X += fr[k] * sv[k]; }
  }
  R Y[4], Ysq = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) { Y[k] = fr[k] - X * sv[k]; Ysq += Y[k] * Y[k]; }
  R Hf = 0, Gf = 0, HY = 0, GY = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) { Hf += Hv[k] * sv[k]; Gf += G[k] * sv[k]; HY += Hv[k] * Y[k]; GY += G[k] * Y[k]; }
  R b4 = (R)0.25 * lam12;
  R b3 = (R)0.25 * (Hf * lore + Gf * loim);
  R b2 = (R)0.5 * msq + (R)3 + (R)0.5 * Ysq * lam12 + (R)0.25 * (HY * lore + GY * loim);
  R b1 = -F + (R)0.25 * Ysq * (Hf * lore + Gf * loim);
  b2 += (R)0.5 * Hsq * (R)cp.lam3 + (R)0.25 * (R)cp.lam4 * (Hf * Hf + Gf * Gf) +
        (R)0.25 * (R)cp.lam5re * (Hf * Hf - Gf * Gf) - (R)0.5 * (R)cp.lam5im * Gf * Hf;
  b1 += (R)0.5 * Hf * (HY * (R)cp.lam4 + HY * (R)cp.lam5re - GY * (R)cp.lam5im) +
        (R)0.5 * Gf * (GY * (R)cp.lam4 - GY * (R)cp.lam5re - HY * (R)cp.lam5im);
  R Xn = polysolve3<R>(b4, b3 + b4 * X, b2 + b3 * X + b4 * X * X, b1 + b2 * X + b3 * X * X + b4 * X * X * X, fallback);
  R dV = (R)4 * b4 * X * X * X + (R)3 * b3 * X * X + (R)2 * b2 * X + b1;
  R dVn = (R)4 * b4 * Xn * Xn * Xn + (R)3 * b3 * Xn * Xn + (R)2 * b2 * Xn + b1;
  if (mabs(dV / dVn) >= u) {
    st4<R>(php(f, h), i, Q<R>{fr[0] + sv[0] * (Xn - X), fr[1] + sv[1] * (Xn - X), fr[2] + sv[2] * (Xn - X),
                             fr[3] + sv[3] * (Xn - X)});
    return 1;
  }
  return 0;
}

// overrelax_triplet (overrelax.c:137-236); no portal term in B (the
// reference's "#ifdef HIGGS" there is never defined)
// The triplet's staple s = -sum_d [R(U_d(x)) t(x+d) + R(U_d(x-d))^T t(x-d)]:
// with it the local action (localact_triplet, su2u1.c:657-679) is
// t.s + B t^2 + C t^4 (+ the portal a2 phi^2 t^2 / 2), B = 3 + msqT / 2,
// C = b4 / 4, the form overrelax.c:137-236 works with.
template <typename R>
__device__ inline V3<R> staple_triplet(const Fields<R>& f, const Geom& g, const int* c, int i) {
  V3<R> s{(R)0, (R)0, (R)0};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    int xp = shifted(g, c, d, 1), xm = shifted(g, c, d, -1);
    V3<R> r = qrot(ldro4<R>(lk(f, d), i), ldro3(f, xp));
    s.x -= r.x; s.y -= r.y; s.z -= r.z;
    r = qrot(qdag(ldro4<R>(lk(f, d), xm)), ldro3(f, xm));
    s.x -= r.x; s.y -= r.y; s.z -= r.z;
  }
  return s;
}

template <typename R, int CC, typename RNG>
__device__ inline int overrelax_triplet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                        RNG& rng, int* fallback) {
  const R u = rng.uni();
  if constexpr (sizeof(R) == 8)
    return overrelax_triplet_f64(f, cp, i, staple_triplet(f, g, c, i), u, fallback);
  V3<R> s = staple_triplet(f, g, c, i);
  V3<R> t = ld3(f, i);
  R F = msqrt(s.x * s.x + s.y * s.y + s.z * s.z);
  const R iF = (R)1 / F;  // one reciprocal instead of seven divisions
  R X = (t.x * s.x + t.y * s.y + t.z * s.z) * iF;
  R y0 = t.x - X * s.x * iF;
  R y1 = t.y - X * s.y * iF;
  R y2 = t.z - X * s.z * iF;
  R Ysq = y0 * y0 + y1 * y1 + y2 * y2;
  R B = (R)0.5 * (R)cp.msqT + (R)3;
  R C = (R)0.25 * (R)cp.b4;
  R cc = B + (R)2 * Ysq * C;
  R newX = polysolve3<R>(C, C * X, cc + C * X * X, F + cc * X + C * X * X * X, fallback);
  R dV = F + (R)2 * B * X + (R)4 * C * (X * X * X + Ysq * X);
  R dVn = F + (R)2 * B * newX + (R)4 * C * (newX * newX * newX + Ysq * newX);
  if (mabs(dV / dVn) >= u) {
    R k = newX + X;
    st3(f, i, V3<R>{-t.x + k * s.x * iF, -t.y + k * s.y * iF, -t.z + k * s.z * iF});
    return 1;
  }
  return 0;
}

// metro_triplet (metropolis.c:113-143).  The reference evaluates
// localact_triplet before and after the change; in their difference every
// term but t.s and the powers of t^2 cancels, so it is formed directly from
// the staple: dS = (t'-t).s + (t'^2-t^2) (B + C (t'^2+t^2)) (+ portal).  One
// gather of the neighbours instead of two, the field written only on accept.
template <typename R, int CC>
__device__ inline int metro_triplet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    SiteRng<R>& rng) {
  if constexpr (sizeof(R) == 8) return metro_triplet_f64<CC>(f, cp, i, staple_triplet(f, g, c, i), rng);
  const R e0 = rng.uni() - (R)0.5, e1 = rng.uni() - (R)0.5, e2 = rng.uni() - (R)0.5;
  // the decision's uniform is the fourth word of the same generator block,
  // drawn with the proposal (FP64 draws it only when it is needed)
  const R ua = rng.uni();
  V3<R> s = staple_triplet(f, g, c, i);
  V3<R> old = ld3(f, i);
  V3<R> nw = old;
  nw.x += (R)1 * e0;
  nw.y += (R)1 * e1;
  nw.z += (R)1 * e2;
  const R dx = nw.x - old.x, dy = nw.y - old.y, dz = nw.z - old.z;
  const R dsq = dx * (nw.x + old.x) + dy * (nw.y + old.y) + dz * (nw.z + old.z);
  const R ssq = (nw.x * nw.x + nw.y * nw.y + nw.z * nw.z) + (old.x * old.x + old.y * old.y + old.z * old.z);
  R B = (R)0.5 * (R)cp.msqT + (R)3;
  if (NHIGGS > 0) B += (R)0.5 * (R)cp.a2 * doubletsq(ld4<R>(php(f, 0), i));
  const R dS = dx * s.x + dy * s.y + dz * s.z + dsq * (B + (R)0.25 * (R)cp.b4 * ssq);
  if (metro_accept_u(dS, ua)) {
    st3(f, i, nw);
    return 1;
  }
  return 0;
}

// localact_singlet (su2u1.c:688-705)
template <typename R, int CC>
__device__ inline R localact_singlet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i) {
  R S = f.sing[i], res = (R)3 * S * S;
#pragma unroll
  for (int d = 0; d < 3; d++) res -= S * (f.sing[shifted(g, c, d, 1)] + f.sing[shifted(g, c, d, -1)]);
  res += potential_singlet<R, CC>(f, cp, i);
  return res;
}

// overrelax_singlet (overrelax.c:243-285)
template <typename R, int CC, typename RNG>
__device__ inline int overrelax_singlet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                        RNG& rng, int* fallback) {
  const R u = rng.uni();
  R S = f.sing[i];
  R c1 = (R)cp.b1s;
#pragma unroll
  for (int d = 0; d < 3; d++) c1 -= (f.sing[shifted(g, c, d, 1)] + f.sing[shifted(g, c, d, -1)]);
  R c2 = (R)3 + (R)0.5 * (R)cp.msqs;
  R c3 = (R)(1.0 / 3.0) * (R)cp.b3s;
  R c4 = (R)0.25 * (R)cp.b4s;
  if (NHIGGS == 1) {
    R phisq = doubletsq(ld4<R>(php(f, 0), i));
    c1 += (R)0.5 * (R)cp.a1s * phisq;
    c2 += (R)0.5 * (R)cp.a2s * phisq;
  }
  R d0 = c1 + c2 * S + c3 * S * S + c4 * S * S * S;
  R d1 = c2 + c3 * S + c4 * S * S;
  R d2 = c3 + c4 * S;
  R Y = polysolve3<R>(c4, d2, d1, d0, fallback);
  R dV = c1 + (R)2 * c2 * S + (R)3 * c3 * S * S + (R)4 * c4 * S * S * S;
  R dVn = c1 + (R)2 * c2 * Y + (R)3 * c3 * Y * Y + (R)4 * c4 * Y * Y * Y;
  if (mabs(dV / dVn) >= u) {
    f.sing[i] = Y;
    return 1;
  }
  return 0;
}

// metro_singlet (metropolis.c:148-167)
template <typename R, int CC>
__device__ inline int metro_singlet(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                    SiteRng<R>& rng) {
  R old = f.sing[i];
  R a0 = localact_singlet<R, CC>(f, g, cp, c, i);
  f.sing[i] = old + (R)1 * (rng.uni() - (R)0.5);
  R a1 = localact_singlet<R, CC>(f, g, cp, c, i);
  if (metro_accept(a1 - a0, rng)) return 1;
  f.sing[i] = old;
  return 0;
}

// order-parameter contribution of one site (calc_orderparam, multicanonical.c:709-751)
template <typename R>
__device__ inline double orderparam_site(const Fields<R>& f, int op, int i) {
  switch (op) {
    case 2: return (double)tripletsq(ld3(f, i));
    case 3: return (double)doubletsq(ld4<R>(php(f, 0), i)) - (double)tripletsq(ld3(f, i));
    case 1: return (double)doubletsq(ld4<R>(php(f, 0), i));
    case 4: return (double)doubletsq(ld4<R>(php(f, 1), i));
  }
  return 0.0;
}

// ---------------------------------------------------------------------------
// half-sweep kernels
// ---------------------------------------------------------------------------
struct PassArgs {
  Geom g;
  CoupT<double> cpd;  // couplings for FP64 kernels
  CoupT<float> cpf;   // the same for FP32 kernels
  RngKey rk;
  int parity;
  int sub;      // direction for links, doublet index for doublets
  int alg;      // algorithm (links) or forced Metropolis flag (scalars)
  uint32_t pass;
  int t_lo, t_hi;       // site range inside the parity
  void* backup;             // multicanonical backup of the updated field (or null)
  int op;                   // order parameter to reduce (0: none)
  double* partials;         // per-block order-parameter sums (or null)
  unsigned long long* ctr;  // device counters (CTR_COPIES copies)
  int* err;                 // device error flag
};

template <typename R>
__device__ inline const CoupT<R>& coup(const PassArgs& a);
template <>
__device__ inline const CoupT<double>& coup<double>(const PassArgs& a) { return a.cpd; }
template <>
__device__ inline const CoupT<float>& coup<float>(const PassArgs& a) { return a.cpf; }

// MU: the link direction of the pass, a template parameter so that every
// neighbour offset and field pointer of the staple is fixed at compile time
template <typename R, int CC, int MU, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_link(Fields<R> f, PassArgs a) {
  dependent_wait();
  const CoupT<R>& cp = coup<R>(a);
  int t = a.t_lo + (int)blockIdx.x * blockDim.x + threadIdx.x;
  int acc = 0, cap = 0, err = 0;
  if (t < a.t_hi) {
    int c[3];
    site_coords(a.g, a.parity, t, c);
    int i = a.parity * a.g.half + t;
    SiteRng<R> rng(a.rk, *a.rk.sweep, (uint32_t)i, a.pass);
    if (a.alg == ALG_HEATBATH) acc = heatbath<R, CC>(f, a.g, cp, c, i, MU, rng, &cap, &err);
    else acc = metro_link<R, CC>(f, a.g, cp, c, i, MU, rng);
  }
  dependents_go();
  unsigned long long* ctr = ctr_copy(a.ctr, blockIdx.x);
  warp_count(ctr + 1, acc);
  warp_count(ctr + 22, cap);
  if (err) atomicOr(a.err, 1);
}

template <typename R, int CC, int MU, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_u1(Fields<R> f, PassArgs a) {
  dependent_wait();
  const CoupT<R>& cp = coup<R>(a);
  int t = a.t_lo + (int)blockIdx.x * blockDim.x + threadIdx.x;
  int acc = 0;
  if (t < a.t_hi) {
    int c[3];
    site_coords(a.g, a.parity, t, c);
    int i = a.parity * a.g.half + t;
    SiteRng<R> rng(a.rk, *a.rk.sweep, (uint32_t)i, a.pass);
    acc = metro_u1<R, CC>(f, a.g, cp, c, i, MU, rng);
  }
  dependents_go();
  warp_count(ctr_copy(a.ctr, blockIdx.x) + 3, acc);
}

// one parity (or a contiguous block of it) of one doublet / the triplet /
// the singlet; optional multicanonical backup of the old values and block
// sums of the order parameter over the new ones
template <typename R, int CC, int FIELD, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_scalar(Fields<R> f, PassArgs a) {
  dependent_wait();
  const CoupT<R>& cp = coup<R>(a);
  int t = a.t_lo + (int)blockIdx.x * blockDim.x + threadIdx.x;
  int acc = 0, fb = 0;
  double opv = 0.0;
  bool orr = false;
  if (t < a.t_hi) {
    int c[3];
    site_coords(a.g, a.parity, t, c);
    int i = a.parity * a.g.half + t;
    SiteRng<R> rng(a.rk, *a.rk.sweep, (uint32_t)i, a.pass);
    if (FIELD == 0) {
      const int h = a.sub;
      if (a.backup) ((V4<R>*)a.backup)[i] = php(f, h)[i];
      orr = cp.alg_d == ALG_OR && !a.alg;
      if (orr) acc = NHIGGS == 2 ? overrelax_higgs2<R, CC>(f, a.g, cp, c, i, h, rng, &fb)
                                 : overrelax_doublet<R, CC>(f, a.g, cp, c, i, rng, &fb);
      else acc = metro_doublet<R, CC>(f, a.g, cp, c, i, h, rng);
    } else if (FIELD == 1) {
      if (a.backup) {
        R* b = (R*)a.backup;
        b[3 * i] = f.trip[0][i]; b[3 * i + 1] = f.trip[1][i]; b[3 * i + 2] = f.trip[2][i];
      }
      orr = cp.alg_t == ALG_OR && !a.alg;
      if (orr) acc = overrelax_triplet<R, CC>(f, a.g, cp, c, i, rng, &fb);
      else acc = metro_triplet<R, CC>(f, a.g, cp, c, i, rng);
    } else {
      orr = cp.alg_s == ALG_OR && !a.alg;
      if (orr) acc = overrelax_singlet<R, CC>(f, a.g, cp, c, i, rng, &fb);
      else acc = metro_singlet<R, CC>(f, a.g, cp, c, i, rng);
    }
    if (a.partials) opv = orderparam_site<R>(f, a.op, i);
  }
  // counters: doublet OR/Metropolis (+h), triplet, singlet
  int base_or = FIELD == 0 ? 10 + a.sub : (FIELD == 1 ? 15 : 19);
  int base_mt = FIELD == 0 ? 6 + a.sub : (FIELD == 1 ? 13 : 17);
  bool any_or = (FIELD == 0 ? cp.alg_d : (FIELD == 1 ? cp.alg_t : cp.alg_s)) == ALG_OR && !a.alg;
  dependents_go();
  unsigned long long* ctr = ctr_copy(a.ctr, blockIdx.x);
  warp_count(ctr + (any_or ? base_or : base_mt), acc);
  warp_count(ctr + 23, fb);
  if (a.partials) {
    double s = block_sum(opv);
    if (threadIdx.x == 0) a.partials[blockIdx.x] = s;
  }
}

// ---------------------------------------------------------------------------
// Split passes, the FP64 form of small lattices: a site's update by four lanes,
// the same lane of the four warps of a block, which run on the four quarters of
// an SM.  A quarter's FP64 pipe takes a warp instruction in 64 cycles however
// many lanes or warps there are, so a pass of fewer warps of sites than there are
// quarters (608) lasts as long as one site's FP64 instructions.  Each warp takes
// a part of the staple (and of the random numbers' functions); the first goes on
// with the sum.  Sweep + measurement of the fundamental theory, one lane a site
// against four: 16^3 (64 groups of 32 sites) 261 / 213 us.  Two sweeps, us, over the
// groups of 32 sites: fundamental 319 468 / 452, 352 462 / 460, 384 468 / 472, 416
// 467 / 476, 512 482 / 525; adjoint 384 513 / 507, 416 513 / 515; SU(2)xU(1) +
// singlet 384 833 / 812, 448 836 / 832, 480 872 / 914: the line is at 384.
// ---------------------------------------------------------------------------
constexpr int SPLIT_GROUPS = 384;

// draw n of the site's stream
__device__ inline double draw_at(SiteRng<double>& rng, uint32_t n) {
  rng.draw = n & ~1u;
  const double v = rng.uni();
  return (n & 1u) ? rng.uni() : v;
}

// Link heatbath (see heatbath).  Before the barrier: warp w computes one of the
// four products of the Wilson staple; warp 1 the logarithms of the first trial,
// warp 2 the direction drawn after it, warp 3 its cosine and the doublets' term.
// A first trial that is rejected (1-2 %) is followed by the others in warp 0.
template <int CC, int MU>
__global__ void __launch_bounds__(128) k_link_split(Fields<double> f, PassArgs a) {
  using R = double;
  constexpr int N0 = MU == 0 ? 1 : 0, N1 = MU == 2 ? 1 : 2;
  __shared__ double s_st[5][4][32], s_log[2][32], s_cos[32], s_n[3][32];
  __shared__ int s_nd[32];
  dependent_wait();
  const CoupT<R>& cp = coup<R>(a);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = a.t_lo + (int)blockIdx.x * 32 + lane;
  const bool on = t < a.t_hi;
  int c[3];
  site_coords(a.g, a.parity, on ? t : a.t_lo, c);
  const Geom& g = a.g;
  const int i = a.parity * g.half + (on ? t : a.t_lo);
  SiteRng<R> rng(a.rk, *a.rk.sweep, (uint32_t)i, a.pass);
  const int xp = shifted(g, c, MU, 1);
  const int nh = NHIGGS;
  auto put = [&](int k, const Q<R>& q) {
    s_st[k][0][lane] = q.a; s_st[k][1][lane] = q.b; s_st[k][2][lane] = q.c; s_st[k][3][lane] = q.d;
  };
  {
    const int nu = w < 2 ? N0 : N1;
    Q<R> q;
    if ((w & 1) == 0) {
      const int xn = shifted(g, c, nu, 1);
      q = qmul(qmul(ld4<R>(lk(f, nu), xp), qdag(ld4<R>(lk(f, MU), xn))), qdag(ld4<R>(lk(f, nu), i)));
    } else {
      const int xpm = shifted(g, c, MU, 1, nu, -1), xm = shifted(g, c, nu, -1);
      q = qmul(qmul(qdag(ld4<R>(lk(f, nu), xpm)), qdag(ld4<R>(lk(f, MU), xm))), ld4<R>(lk(f, nu), xm));
    }
    put(w, q);
  }
  R oldact = 0;
  Q<R> old{};
  if (w == 0) {
    if (HAS(C_T)) {
      old = ld4<R>(lk(f, MU), i);
      oldact = hop_triplet_fwd_u(f, g, c, i, MU, old);
    }
  } else if (w == 1) {
    const R u0 = rng.uni(), u1 = rng.uni();
    s_log[0][lane] = -log(1.0 - u0);
    s_log[1][lane] = -log(1.0 - u1);
  } else if (w == 2) {
    rng.draw = 4;
    R d = 2, r1 = 0, r2 = 0, r3 = 0;
    int it = 0;
    while ((d > 1.0 || d == 0.0) && it <= 4096) {
      r1 = 2.0 * rng.uni() - 1.0;
      r2 = 2.0 * rng.uni() - 1.0;
      r3 = 2.0 * rng.uni() - 1.0;
      d = r1 * r1 + r2 * r2 + r3 * r3;
      it++;
    }
    const R k = rsqrt(d);
    s_n[0][lane] = r1 * k;
    s_n[1][lane] = r2 * k;
    s_n[2][lane] = r3 * k;
    s_nd[lane] = it > 4096 ? -1 : 4 + 3 * it;  // draws used, -1: none was found
  } else {
    const R cs = mcos2pi(draw_at(rng, 2));
    s_cos[lane] = cs * cs;
    Q<R> m{0.0, 0.0, 0.0, 0.0};
    for (int h = 0; h < nh; h++) {
      Q<R> nphi = ld4<R>(php(f, h), xp);
      if (HAS(C_U1)) nphi = qphase(nphi, a1p(f, MU)[i]);
      m = qadd(m, qmul(nphi, qdag(ld4<R>(php(f, h), i))));
    }
    put(4, m);
  }
  __syncthreads();
  int acc = 0, cap = 0, err = 0;
  if (w == 0 && on) {
    auto get = [&](int k) {
      return Q<R>{s_st[k][0][lane], s_st[k][1][lane], s_st[k][2][lane], s_st[k][3][lane]};
    };
    Q<R> V = qscale(qadd(qadd(get(0), get(1)), qadd(get(2), get(3))), -0.5 * cp.beta);
    if (nh > 0) {
      const Q<R> m = get(4);
      V = Q<R>{V.a - 0.5 * m.a, V.b - 0.5 * m.b, V.c - 0.5 * m.c, V.d - 0.5 * m.d};
    }
    R ia = rsqrt(qsq(V));
    V = qscale(V, -ia);
    ia *= 0.5;
    R d = (s_log[0][lane] * s_cos[lane] + s_log[1][lane]) * ia;
    R r3 = 1.0 - draw_at(rng, 3);
    int trials = 1;
    bool ok = !(r3 * r3 > 1.0 - 0.5 * d);  // a NaN ends the trials, as in heatbath
    while (!ok && trials < 200) {
      const uint32_t n = 4u * (uint32_t)trials;
      const R u0 = draw_at(rng, n), u1 = rng.uni(), cs = mcos2pi(rng.uni());
      r3 = 1.0 - rng.uni();
      d = (-log(1.0 - u0) * (cs * cs) - log(1.0 - u1)) * ia;
      trials++;
      ok = !(r3 * r3 > 1.0 - 0.5 * d);
    }
    R a0 = 1.0 - d;
    if (trials >= 200) {  // the loop's cap, even if the last trial succeeded
      a0 = 1e-9;
      cap = 1;
    }
    R rad = 1.0 - a0 * a0;
    if (!(rad < 0.0)) {
      rad = sqrt(rad);
      R n1 = s_n[0][lane], n2 = s_n[1][lane], n3 = s_n[2][lane];
      int nd = s_nd[lane];
      if (trials > 1) {
        rng.draw = 4u * (uint32_t)trials;
        R q = 2;
        int it = 0;
        while ((q > 1.0 || q == 0.0) && it <= 4096) {
          n1 = 2.0 * rng.uni() - 1.0;
          n2 = 2.0 * rng.uni() - 1.0;
          n3 = 2.0 * rng.uni() - 1.0;
          q = n1 * n1 + n2 * n2 + n3 * n3;
          it++;
        }
        const R k = rsqrt(q);
        n1 *= k;
        n2 *= k;
        n3 *= k;
        nd = it > 4096 ? -1 : 4 * trials + 3 * it;
      }
      if (nd < 0) {
        err = 1;
      } else {
        const Q<R> U = qmul(Q<R>{a0, n1 * rad, n2 * rad, n3 * rad}, qdag(V));
        acc = 1;
        if (HAS(C_T)) acc = draw_at(rng, (uint32_t)nd) < exp(oldact - hop_triplet_fwd_u(f, g, c, i, MU, U));
        if (acc) st4<R>(lk(f, MU), i, U);
      }
    }
  }
  dependents_go();
  if (w == 0) {
    unsigned long long* ctr = ctr_copy(a.ctr, blockIdx.x);
    warp_count(ctr + 1, acc);
    warp_count(ctr + 22, cap);
    if (err) atomicOr(a.err, 1);
  }
}

// a doublet (FIELD 0) or the triplet (1): the six neighbour terms of the staple
// are one, two, two and one of the warps'
template <int CC, int FIELD>
__global__ void __launch_bounds__(128) k_scalar_split(Fields<double> f, PassArgs a) {
  using R = double;
  __shared__ double s_st[3][4][32];
  dependent_wait();
  const CoupT<R>& cp = coup<R>(a);
  const Geom& g = a.g;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = FIELD == 0 ? a.sub : 0;
  const int t = a.t_lo + (int)blockIdx.x * 32 + lane;
  const bool on = t < a.t_hi;
  int c[3];
  site_coords(g, a.parity, on ? t : a.t_lo, c);
  const int i = a.parity * g.half + (on ? t : a.t_lo);
  // the sum of terms k of this warp; k = 2 d forward, 2 d + 1 backward
  Q<R> s{0.0, 0.0, 0.0, 0.0};
  auto term = [&](int d, bool back) {
    const int x = shifted(g, c, d, back ? -1 : 1);
    const Q<R> u = back ? qdag(ld4<R>(lk(f, d), x)) : ld4<R>(lk(f, d), i);
    if (FIELD == 0) {
      Q<R> v = qmul(u, ld4<R>(php(f, h), x));
      if (HAS(C_U1)) v = qphase(v, back ? -a1p(f, d)[x] : a1p(f, d)[i]);
      s = Q<R>{s.a - v.a, s.b - v.b, s.c - v.c, s.d - v.d};
    } else {
      const V3<R> v = qrot(u, ld3(f, x));
      s = Q<R>{0.0, s.b - v.x, s.c - v.y, s.d - v.z};
    }
  };
  if (w == 0) {
    term(0, false);
  } else {
    if (w == 1) { term(0, true); term(1, false); }
    else if (w == 2) { term(1, true); term(2, false); }
    else term(2, true);
    s_st[w - 1][0][lane] = s.a; s_st[w - 1][1][lane] = s.b; s_st[w - 1][2][lane] = s.c; s_st[w - 1][3][lane] = s.d;
  }
  __syncthreads();
  int acc = 0, fb = 0;
  double opv = 0.0;
  const bool orr = (FIELD == 0 ? cp.alg_d : cp.alg_t) == ALG_OR && !a.alg;
  if (w == 0 && on) {
#pragma unroll
    for (int k = 0; k < 3; k++)
      s = Q<R>{s.a + s_st[k][0][lane], s.b + s_st[k][1][lane], s.c + s_st[k][2][lane], s.d + s_st[k][3][lane]};
    SiteRng<R> rng(a.rk, *a.rk.sweep, (uint32_t)i, a.pass);
    if (FIELD == 0) {
      if (a.backup) ((V4<R>*)a.backup)[i] = php(f, h)[i];
      if (!orr) acc = metro_doublet_f64<CC>(f, cp, i, h, s, rng);
      else if (NHIGGS == 2) acc = overrelax_higgs2<R, CC>(f, g, cp, c, i, h, rng, &fb, &s);
      else acc = overrelax_doublet_f64<CC>(f, cp, i, s, rng.uni(), &fb);
    } else {
      if (a.backup) {
        R* b = (R*)a.backup;
        b[3 * i] = f.trip[0][i]; b[3 * i + 1] = f.trip[1][i]; b[3 * i + 2] = f.trip[2][i];
      }
      const V3<R> st{s.b, s.c, s.d};
      if (orr) acc = overrelax_triplet_f64(f, cp, i, st, rng.uni(), &fb);
      else acc = metro_triplet_f64<CC>(f, cp, i, st, rng);
    }
    if (a.partials) opv = orderparam_site<R>(f, a.op, i);
  }
  dependents_go();
  if (w == 0) {
    unsigned long long* ctr = ctr_copy(a.ctr, blockIdx.x);
    warp_count(ctr + (FIELD == 0 ? (orr ? 10 : 6) + a.sub : (orr ? 15 : 13)), acc);
    warp_count(ctr + 23, fb);
  }
  if (a.partials) {
    const double sum = block_sum(opv);
    if (threadIdx.x == 0) a.partials[blockIdx.x] = sum;
  }
}

// order parameter of a whole parity (calc_orderparam)
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_orderparam(Fields<R> f, Geom g, int parity, int op, double* partials) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (t < g.half) v = orderparam_site<R>(f, op, parity * g.half + t);
  double s = block_sum(v);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// restore a block of the parity from the backup if the last check rejected
// (a small grid striding over the block: when the check accepted, which is
// the common case, the launch is over as soon as its few blocks have read
// the flag)
template <typename R, int FIELD>
__global__ void k_muca_restore(Fields<R> f, const MucaDev* m, const void* backup, int h, int lo, int hi) {
  dependent_wait();
  if (m->last_accept) return;
  for (int i = lo + (int)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (int)(gridDim.x * blockDim.x)) {
    if (FIELD == 0) {
      php(f, h)[i] = ((const V4<R>*)backup)[i];
    } else {
      const R* b = (const R*)backup;
      f.trip[0][i] = b[3 * i]; f.trip[1][i] = b[3 * i + 1]; f.trip[2][i] = b[3 * i + 2];
    }
  }
}

// ---------------------------------------------------------------------------
// multicanonical decision (multicanonical.c:337-704, update.c:13-30), one block
// ---------------------------------------------------------------------------
__device__ inline void muca_linearize(MucaDev* w) {
  w->slope[0] = 0;
  w->slope[w->bins + 1] = 0;
  w->b[0] = w->W[0];
  w->b[w->bins + 1] = w->W[w->bins + 1];
  for (int i = 1; i < w->bins + 1; i++) {
    w->slope[i] = (w->W[i + 1] - w->W[i]) / (w->pos[i + 1] - w->pos[i]);
    w->b[i] = w->W[i] - w->slope[i] * w->pos[i];
  }
}
__device__ inline int muca_whichbin(const MucaDev* w, double val) {
  if (val < w->min) return 0;
  if (val >= w->max) return w->bins + 1;
  int bmin = 1, bmax = w->bins;
  while (bmin <= bmax) {
    int bin = bmin + (bmax - bmin) / 2;
    double cur = w->pos[bin], nxt = w->pos[bin + 1];
    if ((val < nxt && val > cur) || (fabs(val - cur) < 1e-12)) return bin;
    if (val > cur) bmin = bin + 1;
    else bmax = bin - 1;
  }
  return w->bins;
}
__device__ inline double muca_get_weight(const MucaDev* w, double val) {
  if (val >= w->max) return w->b[w->bins + 1];
  if (val < w->min) return w->b[0];
  int bin = muca_whichbin(w, val);
  if (bin >= w->bins + 1) return w->b[w->bins + 1];
  return w->b[bin] + w->slope[bin] * val;
}
__device__ inline void muca_accumulate(MucaDev* w, double val) {
  int bin = muca_whichbin(w, val);
  if (bin == 0) {
    double dmin = w->pos[2] - w->pos[1];
    if (val < w->pos[1] - 0.5 * dmin) return;
    bin += 1;
  } else if (bin < w->bins + 1) {
    if (val - w->pos[bin] > w->pos[bin + 1] - val) bin = bin + 1;
  } else {
    double dmax = w->pos[w->bins + 1] - w->pos[w->bins];
    if (val > w->pos[w->bins + 1] + 0.5 * dmax) return;
  }
  if (w->mode == 1) {
    w->hits[bin] += 5;
    if (bin > 1) w->hits[bin - 1] += 3;
    if (bin > 2) w->hits[bin - 2] += 1;
    if (bin < w->bins) w->hits[bin + 1] += 3;
    if (bin < w->bins - 1) w->hits[bin + 2] += 1;
  } else if (w->mode == 2) {
    w->hits[bin]++;
    w->hgram[bin] += exp(muca_get_weight(w, val));
  }
}
__device__ inline void muca_update_fast(MucaDev* w) {
  int first = -1;
  double delta = 0.0;
  for (int i = 0; i < w->bins + 2; i++) {
    if (w->pos[i] >= w->wrk_min && w->wrk_max >= w->pos[i]) {
      if (first < 0) first = i;
      delta = (w->hits[i] - w->hits[first]) * w->delta / ((double)w->bins);
      w->W[i] += delta;
    } else if (w->wrk_max < w->pos[i]) {
      w->W[i] += delta;
    }
  }
  w->W[0] = w->W[1];
  w->W[w->bins + 1] = w->W[w->bins];
  muca_linearize(w);
  int tunnel = 0;
  if (w->last_max && w->hits[1] > 0) { w->last_max = 0; tunnel = 1; }
  else if (!w->last_max && w->hits[w->bins] > 0) { w->last_max = 1; tunnel = 1; }
  if (tunnel) w->delta /= 1.5;
  for (int i = 0; i < w->bins + 2; i++) w->hits[i] = 0;
}
__device__ inline void muca_update_slow(MucaDev* w) {
  int n = w->bins + 2;
  double* wold = w->wold;
  for (int i = 0; i < n; i++) wold[i] = w->W[i];
  double dmin = w->pos[2] - w->pos[1];
  w->hgram[1] /= dmin;
  for (int i = 2; i < w->bins + 1; i++) w->hgram[i] /= (w->pos[i + 1] - w->pos[i - 1]);
  int first = -1, last = -1, hits_min = 8;
  for (int i = 1; i < w->bins + 1; i++) {
    if (w->pos[i] >= w->wrk_min && w->wrk_max >= w->pos[i]) {
      if (first < 0) { first = i; continue; }
      w->nsum[i] += w->hits[i];
      int gg = 0;
      if (w->hits[i] >= hits_min && w->hits[i - 1] >= hits_min) {
        gg = w->hits[i] + w->hits[i - 1];
      } else {
        w->W[i] = wold[i] - wold[i - 1] + w->W[i - 1];
        continue;
      }
      long long gsum_new = w->gsum[i] + gg;
      double ln = w->hgram[i - 1] / w->hgram[i];
      ln = -1.0 * gg * log(ln);
      w->W[i] = w->W[i - 1] + ((wold[i] - wold[i - 1]) * w->gsum[i] + ln) / ((double)gsum_new);
      w->gsum[i] = gsum_new;
    } else if (w->wrk_max < w->pos[i]) {
      if (last < 0) last = i - 1;
      w->W[i] += w->W[last] - wold[last];
    }
  }
  for (int i = 0; i < n; i++) { w->hits[i] = 0; w->hgram[i] = 0.0; }
  w->W[0] = w->W[1];
  w->W[w->bins + 1] = w->W[w->bins];
  for (int i = 0; i < n; i++) wold[i] = w->W[i];
  double corr = 0.0;
  if (first < 1) {  // no bin inside the work range: nothing to overcorrect
    muca_linearize(w);
    return;
  }
  if (first == 1) dmin = w->pos[first + 1] - w->pos[first];
  else dmin = w->pos[first + 1] - w->pos[first - 1];
  for (int i = first + 1; i < w->bins + 1; i++) {
    if (i <= last) {
      double diff1 = w->pos[i + 1] - w->pos[i - 1];
      corr = 2.0 * log((dmin / diff1) * w->nsum[i] / w->nsum[first]);
    }
    w->W[i] += corr;
  }
  w->W[0] = w->W[1];
  w->W[w->bins + 1] = w->W[w->bins];
  muca_linearize(w);
  for (int i = 0; i < n; i++) w->W[i] = wold[i];
}

// muca_check (update.c:13-30) once the parity's order parameter `tot` is
// known, by a whole block (every thread calls it; blockDim.x >= 2): weight
// difference, global draw (site 0xffffffff, block = check), accept/reject,
// hits and weight recursion.  The weights of the new and the old value
// (get_weight, multicanonical.c:350-379) are looked up with the bins tested
// by all threads at once -- one pass of independent loads instead of a
// binary search of dependent ones, which on the critical path of every
// check cost more than the update itself.  The bin found is the one the
// reference's binary search (whichbin, multicanonical.c:671-704) returns:
// the unique bin with pos[b] < val < pos[b+1]; a value within 1e-12 of a bin
// edge (where the search may stop at either neighbour) or in no bin takes
// the sequential search.  `sweep` is the chain's sweep number (the global
// draw's counter); the decision (1 accept) is returned to every thread.
// What the decision reads of the weight besides the bins it searches, and
// this thread's first bin k = 1 + threadIdx.x (pos[k], pos[k + 1], b[k],
// slope[k]) -- loaded by the deciding block while it still sums the order
// parameter, so that the decision itself waits on no global load in the
// common case (a value strictly inside a bin of the first blockDim.x)
struct MucaPre {
  double pv0, pv1, mn, mx;
  int bins, mode;
  double cur, nxt, bk, sk;
};
__device__ inline MucaPre muca_preload(const MucaDev* w) {
  MucaPre p;
  p.pv0 = w->param_value[0];
  p.pv1 = w->param_value[1];
  p.mn = w->min;
  p.mx = w->max;
  p.bins = w->bins;
  p.mode = w->mode;
  p.cur = p.nxt = p.bk = p.sk = 0.0;
  const int k = 1 + (int)threadIdx.x;
  if (k <= p.bins) {
    p.cur = w->pos[k];
    p.nxt = w->pos[k + 1];
    p.bk = w->b[k];
    p.sk = w->slope[k];
  }
  return p;
}
// muca_decision: the decision alone, which changes nothing, so that several
// blocks may make it; muca_commit: its consequences, by one thread.
struct MucaDecision {
  int accept;
  double tot, old, nw;
};
__device__ inline MucaDecision muca_decision(const MucaDev* w, const MucaPre& pre, double tot, int parity,
                                             const RngKey& rk, uint32_t pass, uint32_t check, uint32_t sweep) {
  __shared__ int s_bin[2], s_fuzzy[2], s_accept;
  __shared__ double s_W[2];
  const int bins = pre.bins;
  const double old = pre.pv0 + pre.pv1;
  const double nw = tot + (parity ? pre.pv0 : pre.pv1);
  if (threadIdx.x < 2) {
    s_bin[threadIdx.x] = -1;
    s_fuzzy[threadIdx.x] = 0;
  }
  __syncthreads();
  for (int k = 1 + (int)threadIdx.x; k <= bins; k += (int)blockDim.x) {
    const bool first = k == 1 + (int)threadIdx.x;
    const double cur = first ? pre.cur : w->pos[k], nxt = first ? pre.nxt : w->pos[k + 1];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const double v = j ? old : nw;
      if (v < nxt && v > cur) s_bin[j] = k;
      if (fabs(v - cur) < 1e-12 || fabs(v - nxt) < 1e-12) s_fuzzy[j] = 1;
    }
  }
  __syncthreads();
  // W = b[bin] + slope[bin] v (get_weight): by the thread that holds the bin,
  // or with loads by thread j for the other cases
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const double v = j ? old : nw;
    const bool inside = !(v >= pre.mx) && !(v < pre.mn);
    const bool direct = inside && s_bin[j] >= 1 && !s_fuzzy[j] && s_bin[j] <= (int)blockDim.x;
    if (direct && s_bin[j] == 1 + (int)threadIdx.x) s_W[j] = pre.bk + pre.sk * v;
    if (!direct && (int)threadIdx.x == j) {
      double W;
      if (v >= pre.mx) W = w->b[bins + 1];
      else if (v < pre.mn) W = w->b[0];
      else {
        const int bin = (s_bin[j] < 0 || s_fuzzy[j]) ? muca_whichbin(w, v) : s_bin[j];
        W = bin >= bins + 1 ? w->b[bins + 1] : w->b[bin] + w->slope[bin] * v;
      }
      s_W[j] = W;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = philox_uniform53(rk.k0, rk.k1, GLOBAL_SITE, pass, check, sweep, rk.chain, 0);
    s_accept = exp(-(s_W[0] - s_W[1])) > u ? 1 : 0;
  }
  __syncthreads();
  return MucaDecision{s_accept, tot, old, nw};
}
__device__ inline void muca_commit(MucaDev* w, const MucaPre& pre, const MucaDecision& d, int parity,
                                   unsigned long long* ctr) {
  w->param_value[parity] = d.tot;
  if (pre.mode != 0) {
    muca_accumulate(w, d.accept ? d.nw : d.old);
    w->muca_count++;
    if (w->muca_count % w->update_interval == 0) {
      if (pre.mode == 1) muca_update_fast(w);
      else if (pre.mode == 2) muca_update_slow(w);
      w->muca_count = 0;
      w->weight_updates++;
    }
    // the recursion may have changed the other parity's value: read it back
    if (!d.accept) w->param_value[parity] = d.old - w->param_value[1 - parity];
  } else if (!d.accept) {
    w->param_value[parity] = d.old - (parity ? pre.pv0 : pre.pv1);
  }
  w->last_accept = d.accept;
  // fire-and-forget adds: this thread alone writes the chain's counters here
  atomicAdd(ctr + 20, 1ull);
  atomicAdd(ctr + 21, (unsigned long long)d.accept);
}
// both, by a block that decides alone; the decision is returned to every thread
__device__ inline int muca_decide_block(MucaDev* w, const MucaPre& pre, double tot, int parity, const RngKey& rk,
                                        uint32_t pass, uint32_t check, uint32_t sweep, unsigned long long* ctr) {
  const MucaDecision d = muca_decision(w, pre, tot, parity, rk, pass, check, sweep);
  if (threadIdx.x == 0) muca_commit(w, pre, d, parity, ctr);
  __syncthreads();
  return d.accept;
}

// sum of x[0..n) by the block's first 64 threads (blockDim.x >= 64) in a
// fixed order -- lane l adds x[l], x[l + 64], ..., then a tree over the 64
// lane sums -- valid in thread 0.  The loads bypass L1: the values were
// written by other blocks of the same launch.
__device__ inline double fixed_sum64(const double* x, int n) {
  __shared__ double red[64];
  if (threadIdx.x < 64) {
    // lane k adds x[k], x[k + 64], ... in that order; the loads are issued
    // sixteen at a time
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += 64 * 16) {
      double t[16];
#pragma unroll
      for (int j = 0; j < 16; j++) t[j] = k + 64 * j < n ? __ldcg(x + k + 64 * j) : 0.0;
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (k + 64 * j < n) v += t[j];
    }
    red[threadIdx.x] = v;
  }
  __syncthreads();
#pragma unroll
  for (int h = 32; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  return red[0];
}

// whether this block, which has read all it needs, is the last of n to say so
// (the count is put back for the next launch)
__device__ inline bool last_to_arrive(unsigned* arrive, unsigned n) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(arrive, 1u) == n - 1;
    if (s_last) *arrive = 0;
  }
  __syncthreads();
  return s_last != 0;
}

// The multicanonical check of a whole parity, in one launch after the update:
// every block adds the update's block sums (a fixed order, the same value in
// each) and makes the decision, which changes nothing; its share of a rejected
// half goes back from the backup; the block that arrives last, when all have
// read the weight, commits the decision.  Deciding inside the update -- a fence
// and two levels of arrivals in every one of its blocks -- made the 96^3 doublet
// half-sweep 35 us, with a restore launch of 3.4 to follow; it takes 23 without,
// and this launch 11.
constexpr int MUCA_FINISH_BLOCKS = SMS;
template <typename R, int FIELD>
__global__ void __launch_bounds__(256) k_muca_finish(Fields<R> f, MucaDev* w, const double* partials, int np,
                                                     double vol, int parity, RngKey rk, uint32_t pass, uint32_t check,
                                                     unsigned long long* ctr, const void* backup, int h, int lo, int hi,
                                                     unsigned* arrive) {
  dependent_wait();
  const MucaPre pre = muca_preload(w);
  double v = 0.0;
  for (int k = threadIdx.x; k < np; k += 256 * 16) {  // sixteen loads at a time
    double t[16];
#pragma unroll
    for (int j = 0; j < 16; j++) t[j] = k + 256 * j < np ? partials[k + 256 * j] : 0.0;
#pragma unroll
    for (int j = 0; j < 16; j++) v += t[j];
  }
  __shared__ double s_tot;
  v = block_sum(v);
  if (threadIdx.x == 0) s_tot = v / vol;
  __syncthreads();
  const MucaDecision d = muca_decision(w, pre, s_tot, parity, rk, pass, check, *rk.sweep);
  if (!d.accept)
    for (int i = lo + (int)(blockIdx.x * 256 + threadIdx.x); i < hi; i += (int)(gridDim.x * 256)) {
      if (FIELD == 0) {
        php(f, h)[i] = ((const V4<R>*)backup)[i];
      } else {
        const R* b = (const R*)backup;
        f.trip[0][i] = b[3 * i]; f.trip[1][i] = b[3 * i + 1]; f.trip[2][i] = b[3 * i + 2];
      }
    }
  if (last_to_arrive(arrive, gridDim.x) && threadIdx.x == 0) muca_commit(w, pre, d, parity, ctr);
}

#ifdef SU2_WITH_GLOBAL
// muca_check (update.c:13-30) as a kernel of its own, for checks that cover
// part of a parity: the partial sums added in a fixed order, then the
// decision.  One block.
__global__ void k_muca_decide(MucaDev* w, const double* partials, int np, double vol, int parity, RngKey rk,
                              uint32_t pass, uint32_t check, unsigned long long* ctr) {
  __shared__ double red[256];
  const MucaPre pre = muca_preload(w);
  double v = 0.0;
  for (int k = threadIdx.x; k < np; k += blockDim.x) v += partials[k];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  muca_decide_block(w, pre, red[0] / vol, parity, rk, pass, check, *rk.sweep, ctr);
}

// calc_orderparam for the host API: store the parity sum
__global__ void k_muca_set_param(MucaDev* w, const double* partials, int np, double vol, int parity) {
  __shared__ double red[256];
  double v = 0.0;
  for (int k = threadIdx.x; k < np; k += blockDim.x) v += partials[k];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) w->param_value[parity] = red[0] / vol;
}

#endif  // SU2_WITH_GLOBAL

// ---------------------------------------------------------------------------
// measurements (measure.c:71-243)
// ---------------------------------------------------------------------------
// The projected U(1) links (magfield.c:32-184) and the plaquette angle
// alpha_proj (magfield.c:189-216).  The reference forms each projected link
// Pi(x) U_mu(x) Pi(x+mu), Pi = (1 + n.sigma)/2, n = Sigma/|Sigma| (projector(),
// project_u1()), as a complex 2x2 matrix, multiplies the four of a plaquette
// and takes the argument of the trace.  Pi is the rank-one projector |n><n|
// onto the +1 eigenvector of n.sigma, so the product collapses to
//   tr = z(x,d1) z(x+d1,d2) conj(z(x+d2,d1)) conj(z(x,d2)),
//   z(a,mu) = <n_a| U_mu(a) |n_{a+mu}>,
// the same number (the phase of each |n> cancels around the closed loop),
// from 4 spinors and 4 overlaps instead of 8 projectors and 11 matrix
// products.  Each site's spinor takes the chart that avoids the pole opposite
// to Sigma: (|S| + S3, S1 + i S2) or (S1 - i S2, |S| - S3), normalised.
template <typename R>
struct Spinor {
  R r0, i0, r1, i1;
};
template <typename R>
__device__ inline Spinor<R> proj_spinor(const V3<R>& a) {
  const R m = msqrt(a.x * a.x + a.y * a.y + a.z * a.z);
  Spinor<R> s;
  if (a.z >= 0) {
    const R k = (R)1 / msqrt((R)2 * m * (m + a.z));
    s.r0 = (m + a.z) * k; s.i0 = 0; s.r1 = a.x * k; s.i1 = a.y * k;
  } else {
    const R k = (R)1 / msqrt((R)2 * m * (m - a.z));
    s.r0 = a.x * k; s.i0 = -a.y * k; s.r1 = (m - a.z) * k; s.i1 = 0;
  }
  return s;
}
// z = <va| U |vb>, U = [[a + i d, c + i b], [-c + i b, a - i d]] (the SU(2)
// matrix of the link quaternion, as project_u1 builds it)
template <typename R>
__device__ inline void link_overlap(const Spinor<R>& va, const Q<R>& u, const Spinor<R>& vb, R& zr, R& zi) {
  const R w0r = u.a * vb.r0 - u.d * vb.i0 + u.c * vb.r1 - u.b * vb.i1;
  const R w0i = u.a * vb.i0 + u.d * vb.r0 + u.c * vb.i1 + u.b * vb.r1;
  const R w1r = -u.c * vb.r0 - u.b * vb.i0 + u.a * vb.r1 + u.d * vb.i1;
  const R w1i = -u.c * vb.i0 + u.b * vb.r0 + u.a * vb.i1 - u.d * vb.r1;
  zr = va.r0 * w0r + va.i0 * w0i + va.r1 * w1r + va.i1 * w1i;
  zi = va.r0 * w0i - va.i0 * w0r + va.r1 * w1i - va.i1 * w1r;
}
template <typename R>
__device__ inline R alpha_proj(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i, int d1,
                               int d2) {
  int c1[3];
  shift_coords(g, c, d1, 1, c1);
  const int i1 = shifted(g, c, d1, 1), i2 = shifted(g, c, d2, 1), i12 = shifted(g, c1, d2, 1);
  const Spinor<R> sx = proj_spinor(ld3(f, i)), s1 = proj_spinor(ld3(f, i1)), s2 = proj_spinor(ld3(f, i2)),
                  s12 = proj_spinor(ld3(f, i12));
  R z1r, z1i, z2r, z2i, z3r, z3i, z4r, z4i;
  link_overlap(sx, ld4<R>(lk(f, d1), i), s1, z1r, z1i);
  link_overlap(s1, ld4<R>(lk(f, d2), i1), s12, z2r, z2i);
  link_overlap(s2, ld4<R>(lk(f, d1), i2), s12, z3r, z3i);
  link_overlap(sx, ld4<R>(lk(f, d2), i), s2, z4r, z4i);
  // (z1 z2) conj(z3 z4)
  const R pr = z1r * z2r - z1i * z2i, pi = z1r * z2i + z1i * z2r;
  const R qr = z3r * z4r - z3i * z4i, qi = z3r * z4i + z3i * z4r;
  const R tr = pr * qr + pi * qi, ti = pi * qr - pr * qi;
  return matan2(ti, tr) * msqrt((R)cp.beta);
}

// alpha(x; 0,1), alpha(x; 0,2), alpha(x; 1,2) for every site
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_alpha(Fields<R> f, Geom g, CoupT<R> cp, double* alpha) {
  dependent_wait();
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.V) return;
  int parity = t >= g.half;
  int tp = t - parity * g.half;
  int c[3];
  site_coords(g, parity, tp, c);
  alpha[t] = (double)alpha_proj(f, g, cp, c, t, 0, 1);
  alpha[g.V + t] = (double)alpha_proj(f, g, cp, c, t, 0, 2);
  alpha[2 * g.V + t] = (double)alpha_proj(f, g, cp, c, t, 1, 2);
}

// per-site terms of measure() summed over the block into partials[k][block]
// Sources of the projected U(1) field strengths alpha_proj (magfield.c:189-216)
// of the magnetic charge: planes filled by k_alpha (plane 0 = (0,1), 1 = (0,2),
// 2 = (1,2)), or the projections computed where they are needed.
struct AlphaPlanes {
  const double* a;
  int V;
  template <typename R>
  __device__ double operator()(const Fields<R>&, const Geom&, const CoupT<R>&, const int*, int n, int plane) const {
    return a[plane * V + n];
  }
};
struct AlphaOnTheFly {
  template <typename R>
  __device__ double operator()(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* cn, int n,
                               int plane) const {
    const int d1 = plane == 2 ? 1 : 0, d2 = plane == 0 ? 1 : 2;
    return (double)alpha_proj(f, g, cp, cn, n, d1, d2);
  }
};

// magcharge_cube (magfield.c:262-280): the divergence of the magnetic field
// of the projected U(1) over the cube at site i (coordinates c)
template <typename R, typename AF>
__device__ inline double magcharge_site(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                        const AF& alpha) {
  int c0[3], c1[3], c2[3];
  shift_coords(g, c, 0, 1, c0);
  shift_coords(g, c, 1, 1, c1);
  shift_coords(g, c, 2, 1, c2);
  int n0 = shifted(g, c, 0, 1), n1 = shifted(g, c, 1, 1), n2 = shifted(g, c, 2, 1);
  double q = 0.0;
  double B1 = alpha(f, g, cp, c, i, 2), B2 = alpha(f, g, cp, c0, n0, 2);
  q += B2 - B1;
  B1 = -alpha(f, g, cp, c, i, 1);
  B2 = -alpha(f, g, cp, c1, n1, 1);
  q += B2 - B1;
  B1 = alpha(f, g, cp, c, i, 0);
  B2 = alpha(f, g, cp, c2, n2, 0);
  q += B2 - B1;
  return q;
}

// magcharge_cube with the projections computed here: the cube's 8 corner
// spinors and 12 edge overlaps once each (each edge borders two of the six
// faces), then the six face angles as alpha_proj forms them
template <typename R>
__device__ inline R face_angle(R ar, R ai, R br, R bi, R cr, R ci, R dr, R di, R sqrt_beta) {
  const R pr = ar * br - ai * bi, pi = ar * bi + ai * br;
  const R qr = cr * dr - ci * di, qi = cr * di + ci * dr;
  return matan2(pi * qr - pr * qi, pr * qr + pi * qi) * sqrt_beta;
}
template <typename R>
__device__ inline double magcharge_site(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, const int* c, int i,
                                        const AlphaOnTheFly&) {
  int c0[3], c1[3], c01[3];
  shift_coords(g, c, 0, 1, c0);
  shift_coords(g, c, 1, 1, c1);
  shift_coords(g, c0, 1, 1, c01);
  const int i0 = shifted(g, c, 0, 1), i1 = shifted(g, c, 1, 1), i2 = shifted(g, c, 2, 1);
  const int i01 = shifted(g, c0, 1, 1), i02 = shifted(g, c0, 2, 1), i12 = shifted(g, c1, 2, 1);
  const int i012 = shifted(g, c01, 2, 1);
  const Spinor<R> sx = proj_spinor(ld3(f, i)), s0 = proj_spinor(ld3(f, i0)), s1 = proj_spinor(ld3(f, i1)),
                  s2 = proj_spinor(ld3(f, i2)), s01 = proj_spinor(ld3(f, i01)), s02 = proj_spinor(ld3(f, i02)),
                  s12 = proj_spinor(ld3(f, i12)), s012 = proj_spinor(ld3(f, i012));
  // z(y, mu) = <n_y| U_mu(y) |n_{y+mu}> on the cube's edges
  R x0r, x0i, x1r, x1i, x2r, x2i, a1r, a1i, a2r, a2i, b0r, b0i, b2r, b2i, e0r, e0i, e1r, e1i, f2r, f2i, g1r, g1i,
      h0r, h0i;
  link_overlap(sx, ld4<R>(lk(f, 0), i), s0, x0r, x0i);       // (x, 0)
  link_overlap(sx, ld4<R>(lk(f, 1), i), s1, x1r, x1i);       // (x, 1)
  link_overlap(sx, ld4<R>(lk(f, 2), i), s2, x2r, x2i);       // (x, 2)
  link_overlap(s0, ld4<R>(lk(f, 1), i0), s01, a1r, a1i);     // (x+0, 1)
  link_overlap(s0, ld4<R>(lk(f, 2), i0), s02, a2r, a2i);     // (x+0, 2)
  link_overlap(s1, ld4<R>(lk(f, 0), i1), s01, b0r, b0i);     // (x+1, 0)
  link_overlap(s1, ld4<R>(lk(f, 2), i1), s12, b2r, b2i);     // (x+1, 2)
  link_overlap(s2, ld4<R>(lk(f, 0), i2), s02, e0r, e0i);     // (x+2, 0)
  link_overlap(s2, ld4<R>(lk(f, 1), i2), s12, e1r, e1i);     // (x+2, 1)
  link_overlap(s01, ld4<R>(lk(f, 2), i01), s012, f2r, f2i);  // (x+0+1, 2)
  link_overlap(s02, ld4<R>(lk(f, 1), i02), s012, g1r, g1i);  // (x+0+2, 1)
  link_overlap(s12, ld4<R>(lk(f, 0), i12), s012, h0r, h0i);  // (x+1+2, 0)
  const R sb = msqrt((R)cp.beta);
  // the charge in the field precision (the angles are): a site's terms are
  // combined in R, the volume sums are FP64
  R q = 0;
  // plane (1,2) at x + 0 minus at x
  R B1 = face_angle(x1r, x1i, b2r, b2i, e1r, e1i, x2r, x2i, sb);
  R B2 = face_angle(a1r, a1i, f2r, f2i, g1r, g1i, a2r, a2i, sb);
  q += B2 - B1;
  // plane (0,2): at x minus at x + 1
  B1 = -face_angle(x0r, x0i, a2r, a2i, e0r, e0i, x2r, x2i, sb);
  B2 = -face_angle(b0r, b0i, f2r, f2i, h0r, h0i, b2r, b2i, sb);
  q += B2 - B1;
  // plane (0,1) at x + 2 minus at x
  B1 = face_angle(x0r, x0i, a1r, a1i, b0r, b0i, x1r, x1i, sb);
  B2 = face_angle(e0r, e0i, g1r, g1i, h0r, h0i, e1r, e1i, sb);
  q += B2 - B1;
  return (double)q;
}

// measure_local (measure.c:368-487): per site (storage order) Tr Sigma^2 and
// the magnetic charge in units of 2 pi sqrt(beta) -- an integer up to rounding
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_measure_local(Fields<R> f, Geom g, CoupT<R> cp, double denom,
                                                         double* out) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.V) return;
  int parity = t >= g.half;
  int c[3];
  site_coords(g, parity, t - parity * g.half, c);
  out[2 * (size_t)t] = (double)tripletsq(ld3(f, t));
  out[2 * (size_t)t + 1] = magcharge_site(f, g, cp, c, t, AlphaOnTheFly{}) / denom;
}

// measure_along_z (z_coord.c:206-300): sums over the plane z of phi^2 (first
// doublet), Tr Sigma^2, S and S^2; one block per plane, the plane's sites
// enumerated by the two other coordinates (lower direction fastest) and summed
// in a fixed order.  out[z][4], columns of absent fields zero.
constexpr int ZBLOCK = 256;
template <typename R>
__global__ void __launch_bounds__(ZBLOCK) k_measure_z(Fields<R> f, Geom g, int content, int zdir, double* out) {
  const int z = blockIdx.x;
  const int dlo = zdir == 0 ? 1 : 0, dhi = zdir == 2 ? 1 : 2;
  const int La = g.L[dlo], area = g.V / g.L[zdir];
  const bool h = content & (C_H1 | C_H2), tr = content & C_T, sg = content & C_S;
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k = threadIdx.x; k < area; k += ZBLOCK) {
    int c[3];
    c[zdir] = z;
    c[dlo] = k % La;
    c[dhi] = k / La;
    int i = site_index(g, c[0], c[1], c[2]);
    if (h) m[0] += (double)doubletsq(ld4<R>(f.phi[0], i));
    if (tr) m[1] += (double)tripletsq(ld3(f, i));
    if (sg) {
      R s = f.sing[i];
      m[2] += (double)s;
      m[3] += (double)(s * s);
    }
  }
  __shared__ double sm[ZBLOCK / 32][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    double v = m[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sm[w][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int ww = 0; ww < ZBLOCK / 32; ww++) v += sm[ww][threadIdx.x];
    out[4 * (size_t)z + threadIdx.x] = v;
  }
}

// measure() (measure.c:110-233): the terms of site t (storage index) added to
// m[NSUMS]; per-site quantities in R, sums in FP64
template <typename R, int CC, typename AF>
__device__ inline void measure_site(const Fields<R>& f, const Geom& g, const CoupT<R>& cp, int t, const AF& alpha,
                                    double* m) {
  int parity = t >= g.half;
  int i = t;
  int c[3];
  site_coords(g, parity, t - parity * g.half, c);
  // local_su2wilson (su2u1.c:143-157)
  R wl = 0;
  wl += ((R)1 - (R)0.5 * ptrace(f, g, c, i, 0, 1));
  wl += ((R)1 - (R)0.5 * ptrace(f, g, c, i, 0, 2));
  wl += ((R)1 - (R)0.5 * ptrace(f, g, c, i, 1, 2));
  wl = (R)cp.beta * wl;
  // the site's action in the field precision (its terms are), summed in FP64
  R act = wl;
  m[1] += (double)wl;
  if (SU2_HAS(CC, cp.content, C_U1)) {
    R u1w = local_u1wilson(f, g, cp, c, i);
    act += u1w;
    m[2] += (double)u1w;
  }
  act += higgspotential<R, CC>(f, cp, i);
  const int nh = SU2_HAS(CC, cp.content, C_H2) ? 2 : (SU2_HAS(CC, cp.content, C_H1) ? 1 : 0);
  for (int h = 0; h < nh; h++) {
    R mod = doubletsq(ld4<R>(php(f, h), i));
    R cov = covariant_doublet<R, CC>(f, g, cp, c, i, h);
    act += cov;
    m[3 + 3 * h] += (double)cov;
    m[4 + 3 * h] += (double)mod;
    m[5 + 3 * h] += (double)(mod * mod);
  }
  if (SU2_HAS(CC, cp.content, C_T)) {
    R covt = covariant_triplet(f, g, c, i);
    act += covt;
    V3<R> tr = ld3(f, i);
    R tm = tripletsq(tr);
    if (nh > 0) m[14] += (double)(doubletsq(ld4<R>(php(f, 0), i)) * tm);
    m[12] += (double)tm;
    m[13] += (double)(tm * tm);
    R hs = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) hs += hop_triplet_fwd(f, g, c, i, d);
    m[11] += (double)hs;
    double q = magcharge_site(f, g, cp, c, i, alpha);
    m[15] += q;
    m[16] += fabs(q);
  }
  if (nh == 2) {
    Q<R> h1 = ld4<R>(php(f, 0), i), h2 = ld4<R>(php(f, 1), i);
    m[9] += (double)((R)0.5 * (h1.a * h2.a + h1.b * h2.b + h1.c * h2.c + h1.d * h2.d));
    m[10] += (double)((R)0.5 * (h1.d * h2.a + h1.c * h2.b - h1.b * h2.c - h1.a * h2.d));
  }
  if (SU2_HAS(CC, cp.content, C_S)) {
    R S = f.sing[i];
    R kin = (R)3 * S * S;
    R scov = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      R Sn = f.sing[shifted(g, c, d, 1)];
      kin -= S * Sn;
      scov += S * S - S * Sn;
    }
    act += kin;
    m[17] += (double)scov;
    m[18] += (double)S;
    m[19] += (double)(S * S);
    m[20] += (double)(S * S * S);
    m[21] += (double)(S * S * S * S);
    if (nh == 1) {
      R mod = doubletsq(ld4<R>(php(f, 0), i));
      m[22] += (double)(mod * S);
      m[23] += (double)(mod * S * S);
    }
  }
  m[0] += (double)act;
}

// Whether the content produces sum k, and the sums a compile-time content
// produces, numbered: active_sum<CC>(j) is the j-th of nactive_sums<CC>().
__host__ __device__ constexpr bool sum_active(int k, int content) {
  const int nh = (content & C_H2) ? 2 : ((content & C_H1) ? 1 : 0);
  const bool t = content & C_T, s = content & C_S;
  return k < 2 || (k == 2 && (content & C_U1)) || (k >= 3 && k <= 5 && nh > 0) || (k >= 6 && k <= 10 && nh > 1) ||
         (k >= 11 && k <= 16 && t && (k != 14 || nh > 0)) || (k >= 17 && k <= 21 && s) || (k >= 22 && s && nh == 1);
}
template <int CC>
constexpr int nactive_sums() {
  int n = 0;
  for (int k = 0; k < NSUMS; k++) n += sum_active(k, CC);
  return n;
}
template <int CC>
constexpr int active_sum(int j) {
  for (int k = 0; k < NSUMS; k++)
    if (sum_active(k, CC) && j-- == 0) return k;
  return -1;
}

// Sums of N (a power of two <= 32) values over the warp, each lane left with
// one of them: at every step a lane keeps half of its values, adding the other
// lane's, and hands the other half over, so N values take about N FP64 adds
// instead of the 5 N of a tree per value (an FP64 instruction of a warp holds its
// SM quarter's pipe for 64 cycles here).  Lane l ends with value l / (32 / N).
template <int N, int O>
__device__ inline double warp_sums(const double (&v)[N]) {
  if constexpr (N == 1) {
    double r = v[0];
#pragma unroll
    for (int o = O; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
  } else {
    const bool up = threadIdx.x & O;
    double w[N / 2];
#pragma unroll
    for (int j = 0; j < N / 2; j++) {
      const double keep = up ? v[j + N / 2] : v[j], send = up ? v[j] : v[j + N / 2];
      w[j] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
    return warp_sums<N / 2, O / 2>(w);
  }
}

// sums of m[] over the block (blockDim.x a multiple of 32, at most BLOCK) to
// partials[k * nblocks + block].  The runtime content sums the first 16 values,
// and the others if its fields have any of them (a value that they do not have is
// left out below): one tree per value that it has takes longer from six on.
template <int CC>
__device__ inline void block_sums_out(const double* m, int content, double* partials, int nblocks, int block) {
  constexpr int NA = nactive_sums<CC>();
  constexpr int N = CC == C_GENERIC ? NSUMS : (NA <= 4 ? 4 : (NA <= 8 ? 8 : (NA <= 16 ? 16 : 32)));
  __shared__ double sm[BLOCK / 32][N];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int j = -1;  // this thread's sum: its place in sm[w]
  if constexpr (CC == C_GENERIC) {
    double v[16], u[8];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = m[q];
    const double r = warp_sums<16, 16>(v);
    if (!(lane & 1)) sm[w][lane / 2] = r;
    static_assert(NSUMS == 24, "16 and 8 sums");
    if (content & (C_T | C_S)) {
#pragma unroll
      for (int q = 0; q < 8; q++) u[q] = m[16 + q];
      const double t = warp_sums<8, 16>(u);
      if (!(lane & 3)) sm[w][16 + lane / 4] = t;
    }
    if (threadIdx.x < NSUMS && sum_active(threadIdx.x, content)) j = threadIdx.x;
  } else {
    double v[N];
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = q < NA ? m[active_sum<CC>(q < NA ? q : 0)] : 0.0;
    const double r = warp_sums<N, 16>(v);
    if (lane % (32 / N) == 0) sm[w][lane / (32 / N)] = r;
#pragma unroll
    for (int q = 0; q < NA; q++)
      if (active_sum<CC>(q) == (int)threadIdx.x) j = q;
  }
  __syncthreads();
  if (threadIdx.x < NSUMS) {
    double x = 0.0;
    if (j >= 0)
      for (int ww = 0; ww < (int)blockDim.x / 32; ww++) x += sm[ww][j];
    partials[threadIdx.x * nblocks + block] = x;
  }
}

// Sites per thread of a measurement of V sites: up to MEAS_SPT, which spreads
// the block's sum over many sites, but no more than leaves about eight warps per
// SM (the sum depends on the number, so it is a function of the lattice's own
// volume and precision alone).  With 8 everywhere a 16^3 lattice was 4 blocks.
// FP64, where an SM quarter's warps run one after another: rounded up, so that no
// quarter gets a third warp (64^3 fundamental: 142 us rounded down to 6 sites a
// thread, 115 in 7, 132 in 8).
constexpr int MEAS_SPT = 8;
__host__ __device__ inline int meas_spt(int V, bool f64) {
  constexpr int W = 32 * 8 * SMS;
  const int s = f64 && V > 2 * W ? (V + W - 1) / W : V / W;
  return s < 1 ? 1 : (s > MEAS_SPT ? MEAS_SPT : s);
}
// threads per block: one warp where blocks of BLOCK would leave SMs idle
__host__ __device__ inline int meas_threads(int V) { return V <= 2 * SMS * BLOCK ? 32 : BLOCK; }
inline unsigned meas_blocks(int V, bool f64) {
  const int per = meas_spt(V, f64) * meas_threads(V);
  return (unsigned)((V + per - 1) / per);
}

// measure() over the whole lattice; alpha = the k_alpha planes (triplet
// content) or null.  meas_blocks(V) blocks of meas_threads(V) threads.  The
// runtime content takes its full 8 sites in a loop of that many turns: with the
// number in a register the same loop ran at 178 instead of 118 us for two doublets
// at 96^3, 514 instead of 269 at 128^3.
template <typename R, int CC>
__global__ void __launch_bounds__(BLOCK) k_measure(Fields<R> f, Geom g, CoupT<R> cp, const double* alpha,
                                                   double* partials) {
  dependent_wait();
  double m[NSUMS];
#pragma unroll
  for (int k = 0; k < NSUMS; k++) m[k] = 0.0;
  const AlphaPlanes ap{alpha, g.V};
  const int spt = meas_spt(g.V, sizeof(R) == 8);
  if (CC == C_GENERIC && spt == MEAS_SPT) {
    for (int j = 0; j < MEAS_SPT; j++) {
      int t = ((int)blockIdx.x * MEAS_SPT + j) * BLOCK + threadIdx.x;
      if (t < g.V) measure_site<R, CC>(f, g, cp, t, ap, m);
    }
  } else {
    for (int j = 0; j < spt; j++) {
      int t = ((int)blockIdx.x * spt + j) * (int)blockDim.x + threadIdx.x;
      if (t < g.V) measure_site<R, CC>(f, g, cp, t, ap, m);
    }
  }
  block_sums_out<CC>(m, cp.content, partials, gridDim.x, blockIdx.x);
}

#ifdef SU2_WITH_GLOBAL
// fixed-order sum of partials[NSUMS][np] -> out[NSUMS]; one block per sum
__global__ void k_reduce_partials(const double* partials, int np, double* out) {
  dependent_wait();
  __shared__ double red[256];
  const double* row = partials + (size_t)blockIdx.x * np;
  double v = 0.0;
  for (int b = threadIdx.x; b < np; b += blockDim.x) v += row[b];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}
#endif  // SU2_WITH_GLOBAL

// ---------------------------------------------------------------------------
// gradient flow (gradflow.c:190-414): forces from `in`, Euler step into `out`
// ---------------------------------------------------------------------------
template <typename R, int CC>
__device__ inline void flow_site(const Fields<R>& in, const Fields<R>& out, const Geom& g, const CoupT<R>& cp, R dt,
                                 unsigned long long* first_zero) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.V) return;
  int parity = t >= g.half;
  int i = t;
  int c[3];
  site_coords(g, parity, t - parity * g.half, c);
#pragma unroll
  for (int mu = 0; mu < 3; mu++) {
    // grad_force_link (gradflow.c:190-258)
    Q<R> s = qscale(wilson_staple<R, true>(in, g, c, i, mu), -cp.beta / (R)8);  // `in` is not written
    Q<R> U = ld4<R>(lk(in, mu), i);
    if (HAS(C_T)) {
      V3<R> a1 = ld3(in, i), a2 = ld3(in, shifted(g, c, mu, 1));
      Q<R> r = qmul(qmul(Q<R>{(R)0, a2.x, a2.y, a2.z}, qdag(U)), Q<R>{(R)0, a1.x, a1.y, a1.z});
      s.a -= (-r.a) / (R)4;
      s.b -= (-r.b) / (R)4;
      s.c -= (-r.c) / (R)4;
      s.d -= (-r.d) / (R)4;
    }
    Q<R> m = qmul(U, s);
    R fz[3] = {(R)2 * m.b, (R)2 * m.c, (R)2 * m.d};
    R z[3], mod = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      fz[a] *= (R)4 / cp.beta;
      z[a] = dt * fz[a];
      mod += z[a] * z[a];
    }
    // flow_gauge (gradflow.c:361-401)
    if (mod <= (R)0) {
      // one atomic a warp, and none above the marker: a start without forces
      // otherwise sends 3 V of them to one address, 0.5 ms a step at 64^3
      const unsigned k = (unsigned)(i * 3 + mu);
      if (k == __reduce_min_sync(__activemask(), k) && k < *(volatile unsigned long long*)first_zero)
        atomicMin(first_zero, (unsigned long long)k);
      st4<R>(lk(out, mu), i, U);
      continue;
    }
    mod = msqrt(mod);
    R sm = msin(mod);
    Q<R> u{mcos(mod), sm * z[0] / mod, sm * z[1] / mod, sm * z[2] / mod};
    st4<R>(lk(out, mu), i, qmul(u, U));
  }
  if (HAS(C_T)) {
    // grad_force_triplet (gradflow.c:267-330) and flow_triplet (405-414)
    R res[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      V3<R> r = qrot(ld4<R>(lk(in, d), i), ld3(in, shifted(g, c, d, 1)));
      res[0] -= r.x; res[1] -= r.y; res[2] -= r.z;
      int xm = shifted(g, c, d, -1);
      r = qrot(qdag(ld4<R>(lk(in, d), xm)), ld3(in, xm));
      res[0] -= r.x; res[1] -= r.y; res[2] -= r.z;
    }
    V3<R> tr = ld3(in, i);
    R tv[3] = {tr.x, tr.y, tr.z};
    R ts = tripletsq(tr);
    R hm = NHIGGS > 0 ? doubletsq(ld4<R>(php(in, 0), i)) : (R)0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      res[a] += ((R)6 + (R)cp.msqT + (R)2 * (R)cp.b4 * ts) * tv[a];
      if (NHIGGS > 0) res[a] += (R)cp.a2 * hm * tv[a];
    }
    st3(out, i, V3<R>{tv[0] + dt * (-res[0]), tv[1] + dt * (-res[1]), tv[2] + dt * (-res[2])});
  }
}

// One Euler step
template <typename R, int CC>
__global__ void __launch_bounds__(BLOCK) k_flow(Fields<R> in, Fields<R> out, Geom g, CoupT<R> cp, R dt,
                                                unsigned long long* first_zero) {
  flow_site<R, CC>(in, out, g, cp, dt, first_zero);
  dependents_go();
}

// After a step: links at or after the first zero-force link keep their value
// (the reference's early return in flow_gauge), and the other of the two markers
// is made ready for the next step.  A launch over the whole GPU, since a start
// with no gauge force at all (unit links, no triplet) keeps every link in every
// step: 64^3, 10 steps with measurements, 0.27 ms; with the step's last block
// putting them back by itself 20 ms.  Without a zero force it only looks at the
// marker, most of that under the step's end (64^3, 20 steps: 581 us for the whole
// flow, 606 with the step's blocks counting themselves in, 728 with a launch
// before and one after each step).
constexpr int FIXUP_BLOCKS = 8 * SMS;
template <typename R>
__global__ void __launch_bounds__(256) k_flow_fixup(Fields<R> in, Fields<R> out, Geom g,
                                                    const unsigned long long* first_zero,
                                                    unsigned long long* next_zero) {
  dependent_wait();
  const unsigned t0 = blockIdx.x * 256u + threadIdx.x, n = 3u * (unsigned)g.V;
  if (t0 == 0) *next_zero = ~0ull;
  const unsigned long long fz = *first_zero;
  if (fz >= n) return;
  for (unsigned t = t0; t < n; t += gridDim.x * 256u) {
    if (t < (unsigned)fz) continue;
    const int i = (int)(t / 3), mu = (int)(t - 3u * (unsigned)i);
    lk(out, mu)[i] = lk(in, mu)[i];
  }
}

// ---------------------------------------------------------------------------
// transfers, tables, reunitarisation
// ---------------------------------------------------------------------------
// host AoS FP64 (lattice-file order) <-> device SoA
template <typename R>
__global__ void k_import(Fields<R> f, int V, int kind, int h, const double* src) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  switch (kind) {
    case 0:  // links [V][3][4]
      if (t < V * 3) {
        int i = t / 3;
        int d = (int)(t - i * 3);
        const double* s = src + t * 4;
        st4<R>(lk(f, d), i, Q<R>{(R)s[0], (R)s[1], (R)s[2], (R)s[3]});
      }
      break;
    case 1:  // u1 [V][3]
      if (t < V * 3) {
        int i = t / 3;
        a1p(f, t - i * 3)[i] = (R)src[t];
      }
      break;
    case 2:  // doublet [V][4]
      if (t < V) {
        const double* s = src + t * 4;
        st4<R>(php(f, h), t, Q<R>{(R)s[0], (R)s[1], (R)s[2], (R)s[3]});
      }
      break;
    case 3:  // triplet [V][3]
      if (t < V) st3(f, t, V3<R>{(R)src[3 * t], (R)src[3 * t + 1], (R)src[3 * t + 2]});
      break;
    case 4:  // singlet [V]
      if (t < V) f.sing[t] = (R)src[t];
      break;
  }
}
template <typename R>
__global__ void k_export(Fields<R> f, int V, int kind, int h, double* dst) {
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  switch (kind) {
    case 0:
      if (t < V * 3) {
        int i = t / 3;
        int d = (int)(t - i * 3);
        Q<R> q = ld4<R>(lk(f, d), i);
        double* s = dst + t * 4;
        s[0] = q.a; s[1] = q.b; s[2] = q.c; s[3] = q.d;
      }
      break;
    case 1:
      if (t < V * 3) {
        int i = t / 3;
        dst[t] = a1p(f, t - i * 3)[i];
      }
      break;
    case 2:
      if (t < V) {
        Q<R> q = ld4<R>(php(f, h), t);
        double* s = dst + t * 4;
        s[0] = q.a; s[1] = q.b; s[2] = q.c; s[3] = q.d;
      }
      break;
    case 3:
      if (t < V) {
        V3<R> v = ld3(f, t);
        dst[3 * t] = v.x; dst[3 * t + 1] = v.y; dst[3 * t + 2] = v.z;
      }
      break;
    case 4:
      if (t < V) dst[t] = f.sing[t];
      break;
  }
}

// renormalise every link to unit norm (FP32 form, every `interval` sweeps)
template <typename R>
__global__ void k_reunitarize(Fields<R> f, int V, const uint32_t* sweep, int interval) {
  if (interval <= 0 || (*sweep % (uint32_t)interval) != (uint32_t)(interval - 1)) return;
  int t = (int)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= V * 3) return;
  int i = t / 3;
  int d = (int)(t - i * 3);
  Q<R> q = ld4<R>(lk(f, d), i);
  R n = (R)1 / msqrt(qsq(q));
  st4<R>(lk(f, d), i, qscale(q, n));
}

#undef HAS
#undef NHIGGS

}  // namespace su2
