// Per-cell collision algebra of the bulk dynamics, in registers.
//
// Written from the reference's generic dynamics templates (paths relative to the reference
// project).  The floating-point operation order follows those templates so that the FP64
// kernels, compiled without FMA contraction, reproduce the reference's CPU_SISD results
// built with its DISABLE_CSE feature:
//   moments          lbm<>::computeRho/computeJ/computeRhoU   src/dynamics/lbm.h:289-330
//   forced velocity  momenta::ForcedMomentum::computeU        src/dynamics/momenta/elements.h:1600-1608
//   equilibrium      equilibrium<>::secondOrder               src/dynamics/lbm.h:50-64
//   BGK              collision::BGK::apply                    src/dynamics/collision.h:68-78
//   TRT              collision::TRT::apply                    src/dynamics/collision.h:393-416
//   Smagorinsky      SmagorinskyEffectiveOmega                src/dynamics/collisionLES.h:59-89
//                    Pi^neq: lbm<>::computeStress lbm.h:333-352, ForcedStress elements.h:1947-1970,
//                    norm momenta/interface.h:164-173
//   Guo forcing      forcing::PlainGuo / forcing::Guo         src/dynamics/forcing.h:35-65, 115-151
//                    lbm<>::addExternalForce                   src/dynamics/lbm.h:568-588
//   bounce-back      collision::Revert                        src/dynamics/collision.h:465-484
//   ConstRhoBGK      collision::ConstRhoBGK::apply            src/dynamics/collision.h:322-351
#pragma once

#include "lbx_desc.cuh"

namespace lbx {

enum Dyn : int {
  DYN_BGK = 1,
  DYN_TRT = 2,
  DYN_SMAGORINSKY = 3,
  DYN_FORCED_BGK = 4,
  DYN_FORCED_SMAGORINSKY = 5,
  DYN_CONST_RHO = 6
};

// Statistics accumulator: {sum rho, sum |u|^2} in FP64, {count, max |u|^2 bits}.
struct StatAcc {
  double sum[2];
  unsigned long long count;
  unsigned long long maxbits;
};

template <typename R>
struct CollisionParams {
  R omega;
  R omega2;  // TRT: relaxation of the antisymmetric part, trt_omega2(omega, magic)
  R smagorinsky;
  R force[3];
  float relax[4];  // FP32 collisions: Relaxation::set
  // ConstRhoBGK: the statistics of the previous step, whose average density is the
  // AVERAGE_RHO parameter (1 while no step has been counted)
  const StatAcc* avgSrc;
};

// The second relaxation frequency of TRT (collision::TRT::apply); the same for every cell, so it is
// found once where the parameters are set.
template <typename R>
__host__ __device__ __forceinline__ R trt_omega2(R omega, R magic) {
  return R(1) / (magic / (R(1) / omega - R(0.5)) + R(0.5));
}

template <int DYN> struct DynTraits {
  static constexpr bool forced = (DYN == DYN_FORCED_BGK || DYN == DYN_FORCED_SMAGORINSKY);
  static constexpr bool smagorinsky = (DYN == DYN_SMAGORINSKY || DYN == DYN_FORCED_SMAGORINSKY);
  static constexpr bool trt = (DYN == DYN_TRT);
};

// Density and velocity of a cell (forced dynamics: u = j/rho + F/2).
template <int Q, typename R, bool FORCED>
__device__ __forceinline__ void moments(const R (&f)[Q], const R* force, R& rho, R (&u)[3]) {
  using D = Desc<Q>;
  rho = R(0);
  static_for<Q>([&](auto I) { rho += f[I]; });
  rho += R(1);
  u[0] = u[1] = u[2] = R(0);
  static_for<Q>([&](auto I) {
    static_for<D::d>([&](auto A) {
      constexpr int c = D::C[I][A];
      if constexpr (c == 1) u[A] += f[I];
      else if constexpr (c == -1) u[A] -= f[I];
    });
  });
  if constexpr (sizeof(R) == 8) {
    static_for<D::d>([&](auto A) { u[A] /= rho; });  // FP64: the reference's exact division
  } else {
    const R inv = R(1) / rho;  // FP32 collision: one division, within the FP32 tolerance
    static_for<D::d>([&](auto A) { u[A] *= inv; });
  }
  if constexpr (FORCED) {
    static_for<D::d>([&](auto A) { u[A] += force[A] * R(0.5); });
  }
}

// c_i . u accumulated over the non-zero components in axis order (the reference loop adds
// c*u for every axis; the zero terms do not change the rounded sum).
template <int Q, int I, typename R>
__device__ __forceinline__ R c_dot(const R (&u)[3]) {
  using D = Desc<Q>;
  R cu = R(0);
  static_for<D::d>([&](auto A) {
    constexpr int c = D::C[I][A];
    if constexpr (c == 1) cu += u[A];
    else if constexpr (c == -1) cu -= u[A];
  });
  return cu;
}

// f_i^eq - w_i (second order).  FP64 keeps the reference's operation sequence (no fused
// operations: the FP64 unit is built with -fmad=false); the float arithmetic of the FP32 and
// reduced-precision forms uses explicit fused multiply-adds.  Every unit is built without
// implicit contraction, so each kernel variant and launch shape rounds identically.
template <int Q, int I, typename R>
__device__ __forceinline__ R equilibrium(R rho, const R (&u)[3], R uSqr) {
  constexpr R t = weight<Q, R>(I);
  const R cu = c_dot<Q, I>(u);
  if constexpr (sizeof(R) == 8) {
    return rho * t * (R(1) + R(3) * cu + R(4.5) * cu * cu - R(1.5) * uSqr) - t;
  } else {
    const R e = __fmaf_rn(R(4.5) * cu, cu, __fmaf_rn(R(3), cu, R(1) - R(1.5) * uSqr));
    return __fmaf_rn(rho * t, e, -t);
  }
}

// Effective relaxation frequency of the Smagorinsky model.
template <int Q, typename R, bool FORCED>
__device__ __forceinline__ R smagorinsky_omega(const R (&f)[Q], R rho, const R (&u)[3],
                                               const CollisionParams<R>& p) {
  using D = Desc<Q>;
  R us[3] = {u[0], u[1], u[2]};
  if constexpr (FORCED) {
    static_for<D::d>([&](auto A) { us[A] = u[A] - R(0.5) * p.force[A]; });
  }
  R pi[6];
  static_for<D::d>([&](auto A) {
    static_for<D::d>([&](auto B) {
      if constexpr (B >= A) {
        R s = R(0);
        static_for<Q>([&](auto I) {
          constexpr int cab = D::C[I][A] * D::C[I][B];
          if constexpr (cab == 1) s += f[I];
          else if constexpr (cab == -1) s -= f[I];
        });
        s -= rho * us[A] * us[B];
        if constexpr (A == B) s -= R(1) / R(3) * (rho - R(1));
        if constexpr (FORCED) {
          s += R(0.5) * rho * (p.force[A] * us[B] + us[A] * p.force[B]);
        }
        // (xx, xy, xz, yy, yz, zz) in 3D, (xx, xy, yy) in 2D
        constexpr int ip = A * D::d - (A * (A - 1)) / 2 + (B - A);
        pi[ip] = s;
      }
    });
  });
  R n2 = pi[0] * pi[0] + R(2) * pi[1] * pi[1] + pi[2] * pi[2];
  if constexpr (D::d == 3) {
    n2 += pi[2] * pi[2] + pi[3] * pi[3] + R(2) * pi[4] * pi[4] + pi[5] * pi[5];
  }
  const R cs = p.smagorinsky;
  const R piNeqNorm = sqrt(n2);
  const R pre = cs * cs * R(3) * R(3) * R(2) * R(1.4142135623730951);
  const R tauMol = R(1) / p.omega;
  const R tauTurb = R(0.5) * (sqrt(tauMol * tauMol + pre / rho * piNeqNorm) - tauMol);
  return R(1) / (tauMol + tauTurb);
}

// ---- FP32 collisions, one cell or two at once ------------------------------------------------
// The arithmetic of the FP32 and 16-bit forms, on a float (one cell) or a float2 (a pair of cells, on
// the packed two-lane instructions of sm_100).  Every operation is an explicitly rounded add,
// multiply or fused multiply-add, and no product is the operand of a separate add (a packed pair of
// those does get fused), so a lane of a pair gets the bits of a single cell: CUDA's packed
// intrinsics round each component as __fadd_rn, __fmul_rn and __fmaf_rn do.
using F2 = float2;
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vrcp(float a) { return 1.f / a; }
__device__ __forceinline__ float vsqrt(float a) { return sqrtf(a); }
__device__ __forceinline__ F2 vadd(F2 a, F2 b) { return __fadd2_rn(a, b); }
// a - b with one rounding, as __fsub_rn: b * (-1) is exact, so the fused form rounds a + (-b) once
__device__ __forceinline__ F2 vsub(F2 a, F2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ F2 vmul(F2 a, F2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ F2 vrcp(F2 a) { return make_float2(1.f / a.x, 1.f / a.y); }
__device__ __forceinline__ F2 vsqrt(F2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }
template <typename V> __device__ __forceinline__ V vset(float a);
template <> __device__ __forceinline__ float vset<float>(float a) { return a; }
template <> __device__ __forceinline__ F2 vset<F2>(float a) { return make_float2(a, a); }

// The weights of the moving directions, one class per number of non-zero components, in units of an
// axis direction's weight t_1: exact powers of two.  With d = 3 omega t_1, N = omega / d.
template <int Q> __host__ __device__ constexpr int weight_class(int i) {
  return (Desc<Q>::C[i][0] != 0) + (Desc<Q>::C[i][1] != 0) + (Desc<Q>::C[i][2] != 0) - 1;
}
template <int Q> struct Weights {
  static constexpr int classes = Q == 27 ? 3 : 2;
  static constexpr float N = Q == 9 ? 3.f : (Q == 19 ? 6.f : 4.5f);      // 1 / (3 t_1)
  static constexpr float rest = Q == 19 ? 6.f : 4.f;                     // t_0 / t_1
  static constexpr float moving = Q == 9 ? 5.f : (Q == 19 ? 12.f : 9.5f);  // (1 - t_0) / t_1
  static __host__ __device__ constexpr float ratio(int k) {
    return k == 0 ? 1.f : (k == 1 ? (Q == 19 ? 0.5f : 0.25f) : 0.0625f);
  }
};

// Coefficients of the FP32 relaxation that conserve what the collision conserves to the last bit the
// format allows: a population keeps a of itself and takes b of its opposite (BGK: b = 0), and the
// equilibrium's even and odd parts enter with d_even, d_odd = 3 omega t_1, taken from the rounded a
// and b, so that a + b + N d_even and a - b + N d_odd are 1.  Rounding omega t_i direction by
// direction instead leaves a factor 1 + 3e-8 on the momentum of every step, which is most of the
// FP32 form's error after some hundred steps.  Against FP64 after 20 steps of a 131 x 150 x 97 D3Q27
// TRT Taylor-Green flow the largest relative error of a population column fell from 5.2e-5 to 1.8e-6
// (with delta in place of rho - 1 below).
struct Relaxation {
  static void set(int q, float omegaF, float magic, bool trt, float (&r)[4]) {
    const double omega = omegaF, omega2 = trt ? trt_omega2(omega, double(magic)) : omega;
    const double n = q == 9 ? 3.0 : (q == 19 ? 6.0 : 4.5);
    r[0] = float(1.0 - 0.5 * (omega + omega2));
    r[1] = float(0.5 * (omega2 - omega));
    r[2] = float((1.0 - (double(r[0]) + double(r[1]))) / n);
    r[3] = float((1.0 - (double(r[0]) - double(r[1]))) / n);
  }
};

// TRT, Smagorinsky and the Guo-forced forms (and BGK, whose pair this describes, where forced).
// Opposite directions i, j share q = (c_i . J)^2
// with J = rho u (the momentum, plus rho F / 2 where forced) and differ in the sign of what is odd in
// c_i.  With delta = rho - 1 (the sum of the stored f - w) and K = delta - 1.5 J^2 / rho the
// equilibrium, less w, is t (K + 4.5 q / rho +- 3 c_i . J); its constant part cancels against the
// stored w and is never formed.  A pair of BGK costs
//   S = omega t (K + 4.5 q / rho),  f_i' = (1 - omega) f_i + S + 3 omega t c_i . J,  f_j' likewise with -,
// six or seven operations on coefficients that the directions of one weight share.  TRT relaxes the
// even part with omega and the odd part with omega2: f_i' = a f_i + b f_j + S + 3 omega2 t c_i . J with
// a = 1 - (omega + omega2) / 2, b = (omega2 - omega) / 2.  Guo's force t rho (1 - omega / 2)
// (3 (c - u) . F + 9 (c . u) (c . F)) adds to the even part -3 u . F (shared by a weight) and
// 9 (1 - omega / 2) t (c . F) (c . J), to the odd part 3 rho (1 - omega / 2) t c . F.
// The 16-bit and D3Q27 forms are bounded by instruction issue (the operation order of the
// reference's templates took 418 instructions a warp for 32 cells of D3Q19 BGK, two and three times
// that for TRT and the forced Smagorinsky form).  At 192^3, default launch shape, FP16 D3Q27:
// TRT 32.2k -> 39.4k MLUPS, forced Smagorinsky 25.8k -> 35.8k; with two cells a thread, which all
// FP32 arithmetic may now pack, FP16 D3Q19 forced Smagorinsky 35.2k -> 55.8k.
template <int Q, int DYN, typename V>
__device__ __forceinline__ void collide_f32(V (&f)[Q], const CollisionParams<float>& p, V& rhoOut, V& uSqrOut) {
  using D = Desc<Q>;
  using T = DynTraits<DYN>;
  using WT = Weights<Q>;
  constexpr int NC = WT::classes;
  V delta = f[0];
  V j[3] = {vset<V>(0.f), vset<V>(0.f), vset<V>(0.f)};
  V pi[6] = {vset<V>(0.f), vset<V>(0.f), vset<V>(0.f), vset<V>(0.f), vset<V>(0.f), vset<V>(0.f)};
  static_for<Q / 2>([&](auto K) {
    constexpr int i = K + 1, jo = D::OPP[i];
    const V s = vadd(f[i], f[jo]), d = vsub(f[i], f[jo]);
    delta = vadd(delta, s);
    static_for<D::d>([&](auto A) {
      constexpr int c = D::C[i][A];
      if constexpr (c == 1) j[A] = vadd(j[A], d);
      else if constexpr (c == -1) j[A] = vsub(j[A], d);
      if constexpr (T::smagorinsky) {
        static_for<D::d>([&](auto B) {
          if constexpr (B >= A) {
            constexpr int cc = D::C[i][A] * D::C[i][B];
            constexpr int ip = A * D::d - (A * (A - 1)) / 2 + (B - A);
            if constexpr (cc == 1) pi[ip] = vadd(pi[ip], s);
            else if constexpr (cc == -1) pi[ip] = vsub(pi[ip], s);
          }
        });
      }
    });
  });
  const V rho = vadd(delta, vset<V>(1.f));
  const V inv = vrcp(rho);
  V a = vset<V>(p.relax[0]), de = vset<V>(p.relax[2]);
  if constexpr (T::smagorinsky) {
    // Pi^neq with the unforced momentum j; n2 = sum of its squared components
    V n2 = vset<V>(0.f);
    static_for<D::d>([&](auto A) {
      const V ja = vmul(j[A], inv);
      static_for<D::d>([&](auto B) {
        if constexpr (B >= A) {
          constexpr int ip = A * D::d - (A * (A - 1)) / 2 + (B - A);
          V s = vfma(vmul(ja, vset<V>(-1.f)), j[B], pi[ip]);
          if constexpr (A == B) s = vfma(delta, vset<V>(-1.f / 3.f), s);
          if constexpr (T::forced) {
            if constexpr (A == B) {
              s = vfma(vset<V>(p.force[A]), j[A], s);
            } else {
              s = vfma(vset<V>(0.5f * p.force[A]), j[B], s);
              s = vfma(vset<V>(0.5f * p.force[B]), j[A], s);
            }
          }
          n2 = vfma(A == B ? s : vmul(s, vset<V>(2.f)), s, n2);
        }
      });
    });
    const float tau = 1.f / p.omega;
    const float pre = p.smagorinsky * p.smagorinsky * 18.f * 1.4142135623730951f;
    const V root = vsqrt(vfma(vmul(vset<V>(pre), inv), vsqrt(n2), vset<V>(tau * tau)));
    // omega = 2 / (tau + root), and the coefficients of Relaxation::set for it
    de = vmul(vrcp(vadd(root, vset<V>(tau))), vset<V>(2.f / WT::N));
    a = vfma(vset<V>(-WT::N), de, vset<V>(1.f));
  }
  if constexpr (T::forced)
    static_for<D::d>([&](auto A) { j[A] = vfma(vset<V>(0.5f * p.force[A]), rho, j[A]); });
  V jj = vmul(j[0], j[0]);
  static_for<D::d - 1>([&](auto A) { jj = vfma(j[A + 1], j[A + 1], jj); });
  const V ju = vmul(jj, inv);  // rho u^2
  const V k0 = vfma(vset<V>(-1.5f), ju, delta);
  const V e1 = vmul(de, vset<V>(1.f / 3.f));  // omega t_1
  V even = vmul(e1, k0);
  V rest = vmul(vfma(vset<V>(-WT::moving), e1, vmul(de, vset<V>(WT::N))), k0);
  const V quad = vmul(vmul(de, vset<V>(1.5f)), inv);  // 4.5 omega t_1 / rho
  V g, h;  // forced: 9 (1 - omega / 2) t_1 and 3 rho (1 - omega / 2) t_1
  if constexpr (T::forced) {
    const V half = vfma(a, vset<V>(0.5f), vset<V>(0.5f));  // 1 - omega / 2
    g = vmul(half, vset<V>(3.f / WT::N));
    h = vmul(vmul(half, vset<V>(1.f / WT::N)), rho);
    V jf = vmul(j[0], vset<V>(p.force[0]));
    static_for<D::d - 1>([&](auto A) { jf = vfma(j[A + 1], vset<V>(p.force[A + 1]), jf); });
    const V hu = vmul(vmul(h, inv), jf);
    even = vsub(even, hu);
    rest = vfma(vset<V>(-WT::rest), hu, rest);
  }
  V ce[NC], cq[NC], cd[NC], cg[NC], ch[NC];
  const V dd = T::trt ? vset<V>(p.relax[3]) : de;
  static_for<NC>([&](auto C) {
    const V r = vset<V>(WT::ratio(C));
    ce[C] = C == 0 ? even : vmul(even, r);
    cq[C] = C == 0 ? quad : vmul(quad, r);
    cd[C] = C == 0 ? dd : vmul(dd, r);
    if constexpr (T::forced) {
      cg[C] = C == 0 ? g : vmul(g, r);
      ch[C] = C == 0 ? h : vmul(h, r);
    }
  });
  f[0] = vfma(T::trt ? vset<V>(p.relax[0] + p.relax[1]) : a, f[0], rest);
  const V b = vset<V>(p.relax[1]);
  static_for<Q / 2>([&](auto K) {
    constexpr int i = K + 1, jo = D::OPP[i], C = weight_class<Q>(i);
    // c_j . J of the opposite direction, whose first non-zero component is positive
    V cj = vset<V>(0.f);
    float cf = 0.f;
    bool first = true;
    static_for<D::d>([&](auto A) {
      constexpr int c = D::C[jo][A];
      if constexpr (c != 0) {
        if (first) cj = c == 1 ? j[A] : vsub(vset<V>(0.f), j[A]);
        else cj = c == 1 ? vadd(cj, j[A]) : vsub(cj, j[A]);
        first = false;
        if constexpr (T::forced) cf = c == 1 ? cf + p.force[A] : cf - p.force[A];
      }
    });
    V even_i, plus, minus;
    if constexpr (T::forced) {
      const V vcf = vset<V>(cf);
      even_i = vfma(vfma(cq[C], cj, vmul(cg[C], vcf)), cj, ce[C]);
      const V odd = vfma(cd[C], cj, vmul(ch[C], vcf));
      plus = vadd(even_i, odd);
      minus = vsub(even_i, odd);
    } else {
      even_i = vfma(cq[C], vmul(cj, cj), ce[C]);
      plus = vfma(cd[C], cj, even_i);
      minus = vfma(vmul(cd[C], vset<V>(-1.f)), cj, even_i);
    }
    const V fi = f[i], fj = f[jo];
    if constexpr (T::trt) {
      f[jo] = vfma(a, fj, vfma(b, fi, plus));
      f[i] = vfma(a, fi, vfma(b, fj, minus));
    } else {
      f[jo] = vfma(a, fj, plus);
      f[i] = vfma(a, fi, minus);
    }
  });
  rhoOut = rho;
  uSqrOut = vmul(ju, inv);
}

// FP32 BGK keeps the operation order that its FP32 and 16-bit runs have had, so that they repeat bit
// for bit (a request of the ensemble near its stability limit amplifies any other rounding); the
// same on a pair as on a cell.
template <int Q, typename V>
__device__ __forceinline__ void collide_bgk(V (&f)[Q], float omega, V& rhoOut, V& uSqrOut) {
  using D = Desc<Q>;
  V rho = f[0];
  static_for<Q - 1>([&](auto I) { rho = vadd(rho, f[I + 1]); });
  rho = vadd(rho, vset<V>(1.f));
  V j[3] = {vset<V>(0.f), vset<V>(0.f), vset<V>(0.f)};
  static_for<Q>([&](auto I) {
    static_for<D::d>([&](auto A) {
      constexpr int c = D::C[I][A];
      if constexpr (c == 1) j[A] = vadd(j[A], f[I]);
      else if constexpr (c == -1) j[A] = vsub(j[A], f[I]);
    });
  });
  const V inv = vrcp(rho);
  V u[3];
  static_for<D::d>([&](auto A) { u[A] = vmul(j[A], inv); });
  V uSqr = vmul(u[0], u[0]);
  static_for<D::d - 1>([&](auto A) { uSqr = vfma(u[A + 1], u[A + 1], uSqr); });
  const V w = vset<V>(omega), keep = vset<V>(1.f - omega);
  const V base = vfma(vset<V>(-1.5f), uSqr, vset<V>(1.f));
  {
    constexpr float t0 = weight<Q, float>(0);
    f[0] = vfma(w, vfma(vmul(rho, vset<V>(t0)), base, vset<V>(-t0)), vmul(f[0], keep));
  }
  static_for<Q / 2>([&](auto K) {
    constexpr int i = K + 1;
    constexpr int jo = D::OPP[i];
    constexpr float t = weight<Q, float>(i);
    V cj = vset<V>(0.f);  // c_i . j over the non-zero components in axis order
    static_for<D::d>([&](auto A) {
      constexpr int c = D::C[i][A];
      if constexpr (c == 1) cj = vadd(cj, j[A]);
      else if constexpr (c == -1) cj = vsub(cj, j[A]);
    });
    const V cu = vmul(cj, inv);
    const V sym = vfma(vmul(rho, vset<V>(t)), vfma(vmul(vset<V>(4.5f), cu), cu, base), vset<V>(-t));
    const V r3t = vmul(rho, vset<V>(3 * t)), m3t = vmul(rho, vset<V>(-3 * t));
    const V plus = vfma(r3t, cu, sym), minus = vfma(m3t, cu, sym);
    f[i] = vfma(w, plus, vmul(f[i], keep));
    f[jo] = vfma(w, minus, vmul(f[jo], keep));
  });
  rhoOut = rho;
  uSqrOut = uSqr;
}

// Two cells (f[k][i], k = 0, 1) of any FP32 collision but ConstRhoBGK, in place.
template <int Q, int DYN>
__device__ __forceinline__ void collide_x2(float (&f)[2][Q], const CollisionParams<float>& p, float (&rhoOut)[2],
                                           float (&usqOut)[2]) {
  F2 g[Q];
  static_for<Q>([&](auto I) { g[I] = make_float2(f[0][I], f[1][I]); });
  F2 rho, usq;
  if constexpr (DYN == DYN_BGK) collide_bgk<Q>(g, p.omega, rho, usq);
  else collide_f32<Q, DYN>(g, p, rho, usq);
  static_for<Q>([&](auto I) {
    f[0][I] = g[I].x;
    f[1][I] = g[I].y;
  });
  rhoOut[0] = rho.x;
  rhoOut[1] = rho.y;
  usqOut[0] = usq.x;
  usqOut[1] = usq.y;
}

// Collide one cell in place.  Returns the cell statistic {rho, |u|^2}.
template <int Q, typename R, int DYN>
__device__ __forceinline__ void collide(R (&f)[Q], const CollisionParams<R>& p, R& rhoOut, R& uSqrOut) {
  using D = Desc<Q>;
  using T = DynTraits<DYN>;
  if constexpr (DYN == DYN_BGK && sizeof(R) == 4) {
    collide_bgk<Q>(f, p.omega, rhoOut, uSqrOut);
    return;
  } else if constexpr (DYN != DYN_CONST_RHO && sizeof(R) == 4) {
    collide_f32<Q, DYN>(f, p, rhoOut, uSqrOut);
    return;
  }
  R rho, u[3];
  moments<Q, R, T::forced>(f, p.force, rho, u);
  R uSqr = R(0);
  static_for<D::d>([&](auto A) { uSqr += u[A] * u[A]; });

  R omega = p.omega;
  if constexpr (T::smagorinsky) omega = smagorinsky_omega<Q, R, T::forced>(f, rho, u, p);

  if constexpr (DYN == DYN_CONST_RHO) {
    // collision::ConstRhoBGK::apply (src/dynamics/collision.h:336-349): the equilibrium part
    // is rescaled by 1 + (1 - <rho>) / rho, which pulls the lattice's average density back to
    // 1; the cell reports rho + (1 - <rho>) to the statistics.
    double avg = 1.0;
    if (p.avgSrc) {
      const unsigned long long cnt = p.avgSrc->count;
      if (cnt) avg = p.avgSrc->sum[0] / double(cnt);
    }
    const R deltaRho = R(1) - R(avg);
    const R ratioRho = R(1) + deltaRho / rho;
    const R keep = R(1) - omega;
    static_for<Q>([&](auto I) {
      constexpr R t = weight<Q, R>(I);
      const R feq = equilibrium<Q, I>(rho, u, uSqr);
      if constexpr (sizeof(R) == 8) f[I] = ratioRho * (feq + t) - t + keep * (f[I] - feq);
      else f[I] = __fmaf_rn(keep, f[I] - feq, __fmaf_rn(ratioRho, feq + t, -t));
    });
    rhoOut = rho + deltaRho;
    uSqrOut = uSqr;
    return;
  }

  if constexpr (T::trt) {
    const R omega2 = p.omega2;
    // pairs (i, opp(i)) for i = 1 .. q/2, plus the rest population
    {
      const R feq0 = equilibrium<Q, 0>(rho, u, uSqr);
      const R fp = R(0.5) * (f[0] + f[0]);
      const R fm = R(0.5) * (f[0] - f[0]);
      const R ep = R(0.5) * (feq0 + feq0);
      const R em = R(0.5) * (feq0 - feq0);
      f[0] -= omega * (fp - ep) + omega2 * (fm - em);
    }
    static_for<Q / 2>([&](auto K) {
      constexpr int i = K + 1;
      constexpr int j = D::OPP[i];
      const R ei = equilibrium<Q, i>(rho, u, uSqr);
      const R ej = equilibrium<Q, j>(rho, u, uSqr);
      const R fi = f[i], fj = f[j];
      const R fpi = R(0.5) * (fi + fj), fmi = R(0.5) * (fi - fj);
      const R fpj = R(0.5) * (fj + fi), fmj = R(0.5) * (fj - fi);
      const R epi = R(0.5) * (ei + ej), emi = R(0.5) * (ei - ej);
      const R epj = R(0.5) * (ej + ei), emj = R(0.5) * (ej - ei);
      f[i] = fi - (omega * (fpi - epi) + omega2 * (fmi - emi));
      f[j] = fj - (omega * (fpj - epj) + omega2 * (fmj - emj));
    });
  } else {
    const R keep = R(1) - omega;
    static_for<Q>([&](auto I) {
      const R feq = equilibrium<Q, I>(rho, u, uSqr);
      f[I] *= keep;
      f[I] += omega * feq;
    });
  }

  if constexpr (T::forced) {
    const R om = rho * (R(1) - omega * R(0.5));
    static_for<Q>([&](auto I) {
      constexpr R t = weight<Q, R>(I);
      const R cu = c_dot<Q, I>(u) * R(9);
      R ft = R(0);
      static_for<D::d>([&](auto A) {
        constexpr int c = D::C[I][A];
        ft += ((R(c) - u[A]) * R(3) + cu * R(c)) * p.force[A];
      });
      ft *= om * t;
      f[I] += ft;
    });
  }
  rhoOut = rho;
  uSqrOut = uSqr;
}

template <int Q, typename R>
__device__ __forceinline__ void revert(R (&f)[Q]) {
  using D = Desc<Q>;
  static_for<Q / 2>([&](auto K) {
    constexpr int i = K + 1;
    constexpr int j = D::OPP[i];
    const R a = f[i];
    f[i] = f[j];
    f[j] = a;
  });
}

}  // namespace lbx
